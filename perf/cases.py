"""The work that users of htree_b200 have it do, as cases that can be timed: inference forwards, training steps (forward
and backward through autograd) and forwards of a query window against a longer key/value cache, over storage types,
head sizes, group sizes and the tree options, from calls of a few hundred positions to the largest configurations.

A case holds the shape (B, T, H, H_kv, D), the storage type, the tree options (CR = compression_rate, TK =
top_k_per_layer, MTN = max_top_nodes), the mode ("fwd", "train" or "window"; a window call has q for the last W positions
only) and how the keys are distributed."""
import numpy as np
import torch

import htree_b200 as ht
from htree_b200 import configs

_DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16, "float16": torch.float16}


def _case(mode, dtype, B, T, H, H_kv, D, CR, TK, MTN, W=0, keys="normal", name=None):
    c = dict(mode=mode, dtype=dtype, B=B, T=T, H=H, H_kv=H_kv, D=D, CR=CR, TK=TK, MTN=MTN, W=W, keys=keys)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a short ragged sequence in a training loop: launches and host work count as much as arithmetic
        _case("train", "bfloat16", 1, 1000, 16, 2, 64, 16, 16, 100, name="train_short"),
        # the smallest benchmark configuration (cfg1): a forward in fp32
        _case("fwd", "float32", 1, 2048, 8, 2, 64, 16, 32, 64, name="fwd_f32_2k"),
        # generation: one new position per sequence against a cache of 16K, a batch of four
        _case("window", "bfloat16", 4, 16384, 32, 2, 128, 16, 64, 128, W=1, name="decode_16k"),
        # an ordinary fp16 training step with groups of 8 heads and a length that is no multiple of anything
        _case("train", "float16", 2, 7777, 32, 4, 128, 16, 32, 512, name="train_f16_8k"),
        # inference prefill, groups of 16 heads (cfg2)
        _case("fwd", "bfloat16", 1, 32768, 32, 2, 128, 16, 64, 128, name="fwd_32k"),
        # keys with clustered, nearly equal scores, eight children per parent (cfg5), in both storage types of that workload
        _case("train", "float32", 2, 16384, 16, 2, 64, 8, 64, 64, keys="clustered", name="train_f32_16k_clustered"),
        _case("train", "bfloat16", 2, 16384, 16, 2, 64, 8, 128, 64, keys="clustered", name="train_16k_clustered"),
        # fp32 training at the head size of the large configurations
        _case("train", "float32", 1, 4096, 16, 2, 128, 16, 32, 256, name="train_f32_d128_4k"),
        # the operator's default options (512 nodes per layer, 8192 at the top): 32-wide heads at the shape of the
        # operator's own correctness runs, and 128-wide heads in inference
        _case("train", "float16", 1, 12000, 16, 4, 32, 16, 512, 8192, name="train_defaults_d32"),
        _case("fwd", "bfloat16", 1, 20000, 16, 1, 128, 16, 512, 8192, name="fwd_defaults_d128"),
        # long-context inference, groups of 8 heads, four pooled levels (cfg4)
        _case("fwd", "bfloat16", 1, 524288, 32, 4, 128, 16, 64, 512, name="fwd_512k"),
        # the headline training step (cfg3)
        _case("train", "bfloat16", 4, 65536, 64, 4, 128, 16, 64, 256, name="train_64k"),
    ]


def _flops(c):
    """Scores of every level that has to choose among more than TK candidates and of the leaves, values of everything
    accumulated; a backward has S, dP, dq, dK and dV over the accumulated candidates."""
    L = len(configs.level_sizes(c["T"], c["CR"], c["MTN"]))
    nc, acc = configs.attend_counts(c["T"], c["CR"], c["TK"], L)
    if c["mode"] == "window":
        nc, acc = nc[:, -c["W"]:], acc[:, -c["W"]:]
    scored = int(nc[0].sum()) + int(np.where(nc[1:] > c["TK"], nc[1:], 0).sum())
    per = 2 * c["D"] * c["H"] * c["B"]
    return per * (scored + int(acc.sum())) + (per * 5 * int(acc.sum()) if c["mode"] == "train" else 0)


def draw(rng):
    """One more case of the same ranges: 200 to 512K positions, one to 16 heads per key/value head, heads of 32, 64 or 128,
    every storage type, the tree options of the listed cases; no more work than the largest of them."""
    most = _flops(_case("train", "bfloat16", 4, 65536, 64, 4, 128, 16, 64, 256))
    while True:
        mode = rng.choice(["fwd", "train", "train", "window"])
        dtype = rng.choice(["bfloat16", "bfloat16", "float16", "float32"])
        D = rng.choice([32, 64, 128, 128])
        G = rng.choice([1, 2, 4, 5, 8, 8, 12, 16, 16])
        H_kv = rng.choice([1, 2, 4])
        B = rng.choice([1, 1, 2, 4])
        T = int(round(200 * 2622 ** rng.random()))                 # 200 .. 524400
        CR = rng.choice([8, 16, 16])
        TK = rng.choice([16, 32, 64, 64, 128, 512])
        MTN = rng.choice([m for m in (64, 128, 256, 512, 8192) if m <= TK * CR])
        W = int(round(min(T, 2048) ** rng.random())) if mode == "window" else 0
        keys = rng.choice(["normal", "normal", "clustered"])
        c = _case(mode, dtype, B, min(T, 524288), G * H_kv, H_kv, D, CR, TK, MTN, W, keys)
        # fp32 and 32-wide heads do fewer operations a second
        if _flops(c) * (30 if dtype == "float32" or D == 32 else 4 if D == 64 or G < 8 else 2) <= most and B * T * G * H_kv * D <= 1 << 30:
            return c


def prepare(case, seed):
    dev, dt = torch.device("cuda"), _DTYPES[case["dtype"]]
    g = torch.Generator(device=dev).manual_seed(seed)
    B, T, H, H_kv, D = (case[n] for n in ("B", "T", "H", "H_kv", "D"))

    def randn(*shape):
        return torch.randn(*shape, generator=g, device=dev, dtype=dt)

    train = case["mode"] == "train"
    Tq = case["W"] if case["mode"] == "window" else T
    q, v, k = randn(B, Tq, H, D), randn(B, T, H_kv, D), randn(B, T, H_kv, D)
    if case["keys"] == "clustered":      # a rank-4 component that all positions share, with coefficients N(0, 3)
        k = (k.float() + (3.0 * randn(B, T, H_kv, 4).float()) @ randn(4, D).float()).to(dt)
    if train:
        q, k, v = (x.requires_grad_(True) for x in (q, k, v))
    return dict(q=q, k=k, v=v, dO=randn(B, T, H, D) if train else None, mode=case["mode"], q_offset=T - Tq,
                options=dict(compression_rate=case["CR"], max_top_nodes=case["MTN"], top_k_per_layer=case["TK"]))


def run(state):
    q, k, v, options = state["q"], state["k"], state["v"], state["options"]
    if state["mode"] == "train":
        out = ht.htree_forward_triton_autograd(q, k, v, **options)
        dq, dk, dv = torch.autograd.grad(out, (q, k, v), state["dO"])
        return {"out": out.detach(), "dq": dq, "dk": dk, "dv": dv}
    if state["mode"] == "window":
        return {"out": ht.htree_forward(q, k, v, _q_offset=state["q_offset"], **options)}
    return {"out": ht.htree_forward(q, k, v, **options)}


def work(case):
    es = 4 if case["dtype"] == "float32" else 2
    kv = 2 * case["B"] * case["T"] * case["H_kv"] * case["D"]
    qo = 2 * case["B"] * (case["W"] if case["mode"] == "window" else case["T"]) * case["H"] * case["D"]
    once = es * (kv + qo)                                  # k, v, q and out
    if case["mode"] == "train":
        once += es * (qo + kv)                             # dO, dq, dk, dv
    return {"bytes": once, "flops": _flops(case)}


def tolerance(case):
    """With the same nodes selected, 16-bit results differ by the rounding of the probabilities, of the half-precision
    rotations and of the results themselves.  In fp32 the sums are good to 1e-5; rotating a query by its distance from the
    key, or both by their own positions, is equally correct, and the two differ by the rounding of the rotary tables'
    angles, which reaches 5e-4 radians at position 8192."""
    return {"rel": 1e-3} if case["dtype"] == "float32" else {"rel": 1e-2}
