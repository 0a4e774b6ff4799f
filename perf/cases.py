"""Timed workloads: what a structure-prediction trunk asks of this library on one GPU.

``listed()`` names the fixed workloads, ``draw(rng)`` samples further ones from the same ranges.
Every case is one of six kinds:

* ``mul`` / ``attn`` - one module-level operator call (bf16, 128 channels), the way a model that
  selects this backend calls it: the pair tensor and its pad mask on the GPU, the residual add
  fused where the caller has one. From a peptide (tens of tokens: launch latency) to a
  thousand-token complex.
* ``trunk`` - a whole 48-block trunk of a small protein in one call, parameters stacked leaf by leaf.
* ``block`` - one complete Pairformer block (pair track, pair transition, single track) in one
  call, from a small protein to the largest complex that runs on one GPU.
* ``stack`` - the four triangle updates, one operator call each, at the other call sites' shapes:
  the float32 trunk, the template stack (64-channel pairs, a few templates per call) and the
  structural refiner (384 channels, 12 heads).
* ``core`` - the bare attention operator on projected q, k, v with additive biases, the contract
  of the fused attention cores it replaces.

Linear kernels are scaled by their fan-in, so that gates and attention weights spread as they do
in a trained model; output projections are N(0, 0.02^2), which keeps the residual stream at the
scale of its input. The trailing tokens are padding, dropped by the mask.
"""

from __future__ import annotations

import math

import torch

from foldjax_b200.pairformer import pairformer_forward, pairformer_layer_forward
from foldjax_b200.triangle import triangle_multiplication_forward
from foldjax_b200.triangle_attention import attention_core, triangle_attention_forward

C_S, HEADS_S = 384, 16  # single track of the Pairformer block


def listed():
    return [
        # a peptide or one small domain: everything is launch latency
        {"name": "attn-n64", "kind": "attn", "n": 64, "pad": 4, "starting": True, "residual": True},
        {"name": "mul-n77", "kind": "mul", "n": 77, "pad": 0, "incoming": True, "residual": False},
        # the whole trunk of a 128-token protein
        {"name": "trunk48-n128", "kind": "trunk", "n": 128, "pad": 7, "blocks": 48},
        # one block: a small protein of odd length, the 1024-token workload, the 3072-token workload
        {"name": "block-n203", "kind": "block", "n": 203, "pad": 0},
        {"name": "block-n1024", "kind": "block", "n": 1024, "pad": 21},
        {"name": "block-n3072", "kind": "block", "n": 3072, "pad": 60},
        # single operators on a mid-size complex: ragged and unpadded, and padded to a round size
        {"name": "mul-n1003", "kind": "mul", "n": 1003, "pad": 0, "incoming": False, "residual": True},
        {"name": "attn-n512", "kind": "attn", "n": 512, "pad": 64, "starting": False, "residual": True},
        # the float32 trunk at the size its tests and the benchmark use
        {"name": "stack-f32-n256", "kind": "stack", "n": 256, "pad": 0, "batch": 1, "f32": True,
         "c_z": 128, "c_hidden": 128, "heads": 4, "head_dim": 32},
        # four templates of a 200-token protein
        {"name": "stack-template-n200", "kind": "stack", "n": 200, "pad": 9, "batch": 4, "f32": False,
         "c_z": 64, "c_hidden": 128, "heads": 4, "head_dim": 16},
        # structural refiner
        {"name": "stack-refiner-n256", "kind": "stack", "n": 256, "pad": 12, "batch": 1, "f32": False,
         "c_z": 384, "c_hidden": 384, "heads": 12, "head_dim": 32},
        # the attention operator alone
        {"name": "core-n384", "kind": "core", "n": 384, "pad": 20},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["mul", "attn", "trunk", "block", "stack", "stack", "core"])
    if kind in ("mul", "attn"):
        n = _log_int(rng, 32, 1280)
        case = {"kind": kind, "n": n, "pad": rng.choice([0, n // 16]),
                "incoming" if kind == "mul" else "starting": rng.random() < 0.5, "residual": rng.random() < 0.7}
    elif kind == "trunk":
        n = _log_int(rng, 48, 256)
        case = {"kind": kind, "n": n, "pad": rng.choice([0, n // 16]), "blocks": 48}
    elif kind == "block":
        n = _log_int(rng, 96, 3000)
        case = {"kind": kind, "n": n, "pad": rng.choice([0, n // 32])}
    elif kind == "stack":
        shape = rng.choice(["f32", "template", "refiner"])
        if shape == "f32":
            n = _log_int(rng, 48, 384)
            case = {"batch": 1, "f32": True, "c_z": 128, "c_hidden": 128, "heads": 4, "head_dim": 32}
        elif shape == "template":
            n = _log_int(rng, 48, 320)
            case = {"batch": rng.randint(1, 4), "f32": False, "c_z": 64, "c_hidden": rng.choice([64, 128]), "heads": 4,
                    "head_dim": 16}
        else:
            n = _log_int(rng, 48, 320)
            case = {"batch": 1, "f32": False, "c_z": 384, "c_hidden": 384, "heads": 12, "head_dim": 32}
        case = {"kind": kind, "n": n, "pad": rng.choice([0, n // 16]), **case}
    else:
        n = _log_int(rng, 48, 640)
        case = {"kind": kind, "n": n, "pad": rng.choice([0, n // 16])}
    return case


# ------------------------------------------------------------------------------- inputs
class _Make:
    """Seeded device tensors; ``lead`` is the leading layer axis of stacked parameters."""

    def __init__(self, seed, dtype, lead=()):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))
        self.dtype, self.lead = dtype, tuple(lead)

    def normal(self, *shape, std=1.0, mean=0.0, dtype=None):
        return (torch.randn(shape, generator=self.g, device="cuda") * std + mean).to(dtype or self.dtype)

    def lin(self, c_in, c_out, std=None):
        return {"kernel": self.normal(*self.lead, c_in, c_out, std=std or c_in ** -0.5)}

    def norm(self, c):
        return {"scale": self.normal(*self.lead, c, std=0.1, mean=1.0), "bias": self.normal(*self.lead, c, std=0.1)}

    def mul(self, c_z=128, c_h=128):
        return {"norm_in": self.norm(c_z), "p_in": self.lin(c_z, 2 * c_h), "g_in": self.lin(c_z, 2 * c_h),
                "norm_out": self.norm(c_h), "p_out": self.lin(c_h, c_z, 0.02), "g_out": self.lin(c_z, c_z)}

    def attn(self, c_z=128, heads=4, head_dim=32):
        hd = heads * head_dim
        return {"layer_norm": self.norm(c_z), "linear": self.lin(c_z, heads),
                "mha": {"linear_q": self.lin(c_z, hd), "linear_k": self.lin(c_z, hd), "linear_v": self.lin(c_z, hd),
                        "linear_g": self.lin(c_z, hd), "linear_o": self.lin(hd, c_z, 0.02)}}

    def transition(self, c):
        return {"norm": self.norm(c), "fc1": self.lin(c, 4 * c), "fc2": self.lin(c, 4 * c), "fc3": self.lin(4 * c, c, 0.02)}

    def block(self):
        proj_q = self.lin(C_S, C_S)
        proj_q["bias"] = self.normal(*self.lead, C_S, std=0.1)
        return {
            "tri_mul_out": self.mul(), "tri_mul_in": self.mul(), "tri_att_start": self.attn(), "tri_att_end": self.attn(),
            "transition_z": self.transition(128), "pre_norm_s": self.norm(C_S),
            "attention": {"proj_q": proj_q, "proj_k": self.lin(C_S, C_S), "proj_v": self.lin(C_S, C_S),
                          "proj_g": self.lin(C_S, C_S), "proj_z_norm": self.norm(128), "proj_z": self.lin(128, HEADS_S),
                          "proj_o": self.lin(C_S, C_S, 0.02)},
            "transition_s": self.transition(C_S),
        }


def _masks(n, pad, batch=1):
    token = torch.ones(batch, n, device="cuda")
    if pad:
        token[:, n - pad:] = 0.0
    return token, (token[:, :, None] * token[:, None, :]).contiguous()


def prepare(case, seed):
    n, kind = case["n"], case["kind"]
    make = _Make(seed, torch.float32 if case.get("f32") else torch.bfloat16, (case["blocks"],) if kind == "trunk" else ())
    token, pair = _masks(n, case["pad"], case.get("batch", 1))
    state = {"case": case, "token": token, "pair": pair}
    if kind == "mul":
        state["params"] = make.mul()
    elif kind == "attn":
        state["params"] = make.attn()
    elif kind in ("trunk", "block"):
        state["params"] = make.block()
        state["s"] = make.normal(1, n, C_S, dtype=torch.float32)
    elif kind == "stack":
        sizes = (case["c_z"], case["heads"], case["head_dim"])
        state["params"] = [make.mul(case["c_z"], case["c_hidden"]), make.mul(case["c_z"], case["c_hidden"]),
                           make.attn(*sizes), make.attn(*sizes)]
    else:  # core: q arrives scaled by 1 / sqrt(32), dropped keys carry -1e9
        q, k, v = (make.normal(1, n, 4, n, 32, std=s) for s in (32 ** -0.5, 1.0, 1.0))
        state.update(q=q, k=k, v=v, bias=make.normal(1, 1, 4, n, n), mask_bias=(1e9 * (pair - 1.0))[:, :, None, None, :])
        return state
    state["z"] = make.normal(case.get("batch", 1), n, n, case.get("c_z", 128))
    return state


# ---------------------------------------------------------------------------------- pass
def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "core":
        return attention_core(state["q"], state["k"], state["v"], state["bias"], state["mask_bias"])
    z, pair, params = state["z"], state["pair"], state["params"]
    if kind == "mul":
        return triangle_multiplication_forward(params, z, pair, "incoming" if case["incoming"] else "outgoing",
                                               residual=z if case["residual"] else None)
    if kind == "attn":
        return triangle_attention_forward(params, z, pair, starting=case["starting"],
                                          residual=z if case["residual"] else None)
    if kind == "block":
        return pairformer_layer_forward(params, state["s"], z, state["token"], pair)
    if kind == "trunk":
        return pairformer_forward(params, state["s"], z, state["token"], pair, num_blocks=case["blocks"])
    z = triangle_multiplication_forward(params[0], z, pair, "outgoing", residual=z)
    z = triangle_multiplication_forward(params[1], z, pair, "incoming", residual=z)
    z = triangle_attention_forward(params[2], z, pair, starting=True, residual=z)
    return triangle_attention_forward(params[3], z, pair, starting=False, residual=z)


# --------------------------------------------------------------------- floor and tolerance
def _mul_flops(n, c_z=128, c_h=128):
    return 2.0 * n**3 * c_h + 2.0 * n**2 * (4 * c_z * c_h + c_h * c_z + c_z * c_z)


def _attn_flops(n, c_z=128, heads=4, head_dim=32):
    hd = heads * head_dim
    return 4.0 * n**3 * hd + 2.0 * n**2 * (5 * c_z * hd + c_z * heads)


def _block_flops(n):
    pair = 2 * _mul_flops(n) + 2 * _attn_flops(n) + 2.0 * n**2 * 3 * 128 * 512
    single = 2.0 * n**2 * 128 * HEADS_S + 4.0 * n**2 * C_S + 2.0 * n * (5 * C_S * C_S + 3 * C_S * 4 * C_S)
    return pair + single


def work(case):
    n, kind = case["n"], case["kind"]
    mask = 4.0 * n * n
    mul_w, attn_w = 2.0 * 128 * 128 * 6, 2.0 * 128 * (128 * 5 + 4)
    if kind == "mul":
        return {"bytes": 2 * n * n * 256.0 + mask + mul_w, "flops": _mul_flops(n)}
    if kind == "attn":
        return {"bytes": 2 * n * n * 256.0 + mask + attn_w, "flops": _attn_flops(n)}
    if kind in ("trunk", "block"):
        blocks = case.get("blocks", 1)
        weights = 2 * mul_w + 2 * attn_w + 2.0 * (3 * 128 * 512 + 128 * HEADS_S + 5 * C_S * C_S + 3 * C_S * 4 * C_S)
        return {"bytes": 2 * n * n * 256.0 + mask + 2 * n * C_S * 4.0 + blocks * weights, "flops": blocks * _block_flops(n)}
    if kind == "core":
        return {"bytes": 4 * n * n * 256.0 + 4 * n * n * 2.0 + mask, "flops": 4.0 * n**3 * 128}
    b, c_z, c_h, heads, hd = (case[k] for k in ("batch", "c_z", "c_hidden", "heads", "head_dim"))
    size = 4.0 if case["f32"] else 2.0
    weights = 2 * size * (5 * c_z * c_h + c_z * c_z) + 2 * size * (5 * c_z * heads * hd + c_z * heads)
    return {"bytes": b * n * n * (2 * c_z * size + 4.0) + weights,
            "flops": b * (2 * _mul_flops(n, c_z, c_h) + 2 * _attn_flops(n, c_z, heads, hd))}


def tolerance(case):
    if case.get("f32"):
        return {"rel": 1e-5}  # float32 sums
    if case["kind"] == "trunk":
        return {"rel": 2e-2}  # 240 bf16 roundings of the residual stream
    return {"rel": 1e-2}  # bf16
