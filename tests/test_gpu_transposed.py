"""The kernels that put candidates on the matrix rows and heads on the columns (operand blocks, selection, accumulation, the
two-pass backward) against the kernels that gather rows, at the sizes where they can go wrong: one position, one position
more or less than a block of children, ragged lengths, 1 / 8 / 9 / 16 heads per group, both branchings, every head size and type."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF, HF, FP = torch.bfloat16, torch.float16, torch.float32


def _inputs(dt, B, T, Hkv, G, D, clustered=False):
    g = torch.Generator(device=DEV).manual_seed(T * 131 + G * 7 + D)
    q, k, v, dO = (torch.randn(B, T, h, D, device=DEV, dtype=dt, generator=g) for h in (Hkv * G, Hkv, Hkv, Hkv * G))
    if clustered:
        k = (k.float() + 3 * torch.randn(B, T, Hkv, 4, device=DEV, generator=g) @ torch.randn(4, D, device=DEV, generator=g)).to(dt)
    return q, k, v, dO


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-20)).item()


@pytest.mark.parametrize("dt,D,CR,G,B,T,TK,MTN", [
    (BF, 128, 16, 16, 1, 1, 16, 64), (BF, 128, 16, 9, 2, 257, 16, 64), (BF, 128, 16, 8, 1, 3001, 32, 128),
    (HF, 128, 8, 16, 1, 1777, 16, 64), (HF, 64, 8, 1, 2, 255, 16, 64), (BF, 64, 16, 16, 1, 1777, 512, 8192),
    (FP, 64, 8, 8, 1, 1777, 16, 64), (FP, 64, 16, 9, 1, 17, 16, 64), (FP, 128, 16, 4, 1, 3001, 32, 64), (FP, 128, 8, 16, 1, 500, 16, 64),
    (HF, 32, 16, 4, 1, 3001, 512, 512), (BF, 32, 8, 12, 1, 1777, 16, 64), (FP, 32, 16, 1, 2, 16, 16, 64)])
def test_forward_and_backward(dt, D, CR, G, B, T, TK, MTN, monkeypatch):
    import htree_b200 as ht
    from htree_b200 import ops
    q, k, v, dO = _inputs(dt, B, T, 2, G, D)
    out, ctx = ht.htree_forward(q, k, v, CR, MTN, TK, _save_for_backward=True)
    assert ctx["layers_v_blk"] is not None, "these sizes are meant to take the operand blocks"
    ref, rctx = ht.htree_forward(q, k, v, CR, MTN, TK, _save_for_backward=True, _force_generic=True)
    alone = ht.htree_forward(q, k, v, CR, MTN, TK)      # inference splits a group over eight warps where there are few groups
    assert torch.equal(alone, out) if B * T * 2 > 296 else _rel(alone, out) < (2e-6 if dt == FP else 4e-3)
    # outputs where the selections agree (16-bit scores have half-precision operands: a few near-ties fall the other way)
    exact = dt == FP or D == 32
    same = torch.stack([(ctx["per_layer_parents"][l] == rctx["per_layer_parents"][l]).all(-1) for l in range(ctx["num_layers"])]).all(0)
    assert same.float().mean().item() >= (1.0 if exact else 0.98)
    rows = same.repeat_interleave(G, -1)
    assert _rel(out[rows], ref[rows]) < (1e-5 if dt == FP else 4e-3)
    # gradients from the same saved state
    ours, gen = ht.htree_backward(dO, q, out, ctx), ht.htree_backward(dO, q, out, ctx, _force_generic=True)
    for a, b in zip(ours, gen):
        # (one position attends to itself alone: P = 1 and dq, dk are zero up to rounding)
        assert (a - b).abs().max().item() < 1e-2 if T == 1 else _rel(a, b) < (1e-5 if exact else 3e-3)
    # several windows of queries instead of one
    monkeypatch.setattr(ops, "BACKWARD_MAX_BYTES", 1 << 22)
    parts = ht.htree_backward(dO, q, out, ctx)
    assert torch.equal(parts[0], ours[0])
    assert T == 1 or max(_rel(a, b) for a, b in zip(parts[1:], ours[1:])) < 1e-5
    torch.cuda.synchronize()
    ops.check_status()


@pytest.mark.parametrize("dt,D,CR,G,B,T,TK,MTN,clustered", [
    (BF, 128, 16, 16, 1, 140, 16, 64, False),      # fewer than 296 groups: eight warps a group
    (BF, 128, 16, 16, 1, 12000, 512, 2048, False), # 752 candidates, more than a level keeps for the last positions only
    (BF, 128, 16, 16, 1, 72000, 512, 8192, False), # 4512 candidates: lists too long for one warp
    (BF, 128, 16, 12, 1, 9001, 32, 256, True), (HF, 128, 8, 8, 1, 9001, 32, 128, False), (BF, 64, 8, 4, 1, 5000, 64, 64, True),
    (HF, 64, 16, 9, 2, 1777, 16, 64, False), (FP, 64, 8, 1, 1, 1777, 16, 64, False), (FP, 64, 16, 16, 1, 5000, 64, 64, True)])
def test_selections_bit_identical(dt, D, CR, G, B, T, TK, MTN, clustered):
    import htree_b200 as ht
    from htree_b200 import ops
    q, k, v, _ = _inputs(dt, B, T, 2, G, D, clustered)
    _, ctx = ht.htree_forward(q, k, v, CR, MTN, TK, _save_for_backward=True)
    gathered = ops.recompute_parents(q, ctx["layers_k"], ctx["layers_v"], ctx["cos_cache"], ctx["sin_cache"], CR, TK, MTN, ctx["scale"], ctx["layers_k_rot"])
    for l, want in gathered.items():
        assert torch.equal(ctx["per_layer_parents"][l], want), f"level {l}"
    w = min(5, T)
    _, cw = ht.htree_forward(q[:, T - w:].contiguous(), k, v, CR, MTN, TK, _q_offset=T - w, _save_for_backward=True)
    for l, want in gathered.items():
        assert torch.equal(cw["per_layer_parents"][l], want[:, T - w:]), f"level {l}, last positions alone"
    torch.cuda.synchronize()
    ops.check_status()


@pytest.mark.parametrize("dt,D,CR,G,T,TK,MTN,W", [
    (BF, 128, 16, 16, 20000, 64, 64, 1), (HF, 64, 16, 8, 9001, 16, 64, 17), (FP, 64, 8, 8, 9001, 32, 128, 3), (HF, 32, 16, 4, 9001, 16, 64, 1),
    (BF, 128, 16, 16, 4000, 16, 64, 125), (BF, 128, 16, 16, 4000, 16, 64, 8),       # either side of 2 * W * TK = parents
    # blocks per query: 8, 4, 2 and 1 (by the room on the chip), 2 (by the chunks of a level); long lists; fp32 of 128 dims; 8 children
    (BF, 128, 16, 16, 20000, 128, 64, 9), (BF, 128, 16, 16, 20000, 128, 64, 18), (BF, 128, 16, 16, 20000, 128, 64, 37),
    (BF, 128, 16, 16, 20000, 128, 64, 38), (BF, 64, 16, 16, 20000, 16, 64, 2), (BF, 128, 16, 4, 30000, 128, 2048, 1),
    # (a thousand values and more: among the 256 of a single head the share bounded below, 1 in 100, is two or three chance roundings)
    (FP, 128, 16, 16, 9001, 128, 128, 5), (BF, 128, 8, 9, 12000, 512, 512, 2)])
def test_few_queries(dt, D, CR, G, T, TK, MTN, W):
    import htree_b200 as ht
    from htree_b200 import ops
    q, k, v, _ = _inputs(dt, 1, T, 2, G, D)
    for sharp in (1, 4):                 # 4: scores spread over 30, so that softmax references move along the walk
        full = ht.htree_forward(q * sharp, k, v, CR, MTN, TK)
        part = ht.htree_forward((q * sharp)[:, T - W:].contiguous(), k, v, CR, MTN, TK, _q_offset=T - W)
        # Sums in another order differ by up to 1e-6 relative (the tensor core truncates its fp32 sums).  A 16-bit result falls on the
        # other side of a rounding boundary with 1e-6 / 2^-8 (bf16; 2^-11: fp16), 1 in 500 at most.  Room for five times that share; at
        # one ulp (2^-7 or 2^-10) each, and values of twice the rms, its 2-norm is 2^-7 * sqrt(1e-2) = 8e-4 or 1e-4.
        want = full[:, T - W:]
        assert _rel(part, want) < (2e-6 if dt == FP else 8e-4 if dt == BF else 1e-4)
        if dt != FP and D > 32:
            assert (part != want).float().mean().item() < 1e-2, "rows depend on how many queries share the call"
    torch.cuda.synchronize()
    ops.check_status()


@pytest.mark.parametrize("dt,D,CR,G,T,TK,MTN,W,zero", [
    (BF, 128, 16, 16, 9001, 32, 128, 3, "q"), (HF, 64, 8, 4, 9001, 64, 64, 40, "k"), (FP, 64, 16, 8, 9001, 32, 64, 2, "q"),
    (BF, 128, 16, 9, 9001, 32, 128, 400, "k"),      # one warp per group
    (BF, 128, 16, 4, 72000, 512, 8192, 600, "q")])  # lists above 4096 candidates
def test_equal_importances(dt, D, CR, G, T, TK, MTN, W, zero):
    """Every candidate but the forced one equally important: the smallest positions are kept, and no search runs."""
    import htree_b200 as ht
    from htree_b200 import ops
    q, k, v, _ = _inputs(dt, 1, T, 2, G, D)
    (q if zero == "q" else k).zero_()
    q = q[:, T - W:].contiguous()
    lists = []
    for generic in (False, True):
        _, ctx = ht.htree_forward(q, k, v, CR, MTN, TK, _q_offset=T - W, _save_for_backward=True, _force_generic=generic)
        lists.append(ctx["per_layer_parents"])
    for l in lists[0]:
        assert torch.equal(lists[0][l], lists[1][l]), f"level {l}"
    torch.cuda.synchronize()
    ops.check_status()


@pytest.mark.parametrize("dt,D,CR,G,T,TK,MTN", [(BF, 128, 16, 16, 3001, 32, 128), (FP, 64, 8, 8, 1777, 16, 64), (HF, 64, 16, 4, 300, 32, 64)])
@pytest.mark.parametrize("compact", [False, True])
def test_malformed_parent_lists(dt, D, CR, G, T, TK, MTN, compact, monkeypatch):
    """A backward whose caller's lists have holes, ids past the end of a level, or more entries than the level has parents reads and
    writes nothing out of range, reports it, and leaves the other queries' gradients as they are."""
    import htree_b200 as ht
    from htree_b200 import ops
    if compact:
        monkeypatch.setattr(ops, "SELECTION_STORAGE", "uint16")
    q, k, v, dO = _inputs(dt, 1, T, 2, G, D)
    out, ctx = ht.htree_forward(q, k, v, CR, MTN, TK, _save_for_backward=True)
    want = ht.htree_backward(dO, q, out, ctx)[0]
    lists = {l: x.clone() for l, x in ctx["per_layer_parents"].items()}
    for bad in range(3):
        ctx["per_layer_parents"] = hurt = {l: x.clone() for l, x in lists.items()}
        rows = torch.arange(T // 2, T, 7, device=DEV)
        leaf, top = hurt[0], hurt[ctx["num_layers"] - 1]
        if bad == 0:                                  # holes, the first entry among them
            leaf[:, rows, 0, 1] = -1
            leaf[:, rows, 1, 0] = -1
        elif bad == 1:                                # past the end (the largest 16-bit id where ids are 16-bit)
            leaf[:, rows, 0, 2] = -2 if compact else 1 << 30
            top[:, rows, 1, 0] = (T + CR - 1) // CR
        else:                                         # as many entries as fit, all of one parent, and a list of none
            leaf[:, rows, 0] = 3
            leaf[:, rows, 1] = -1
        got = ht.htree_backward(dO, q, out, ctx)
        torch.cuda.synchronize()
        assert all(x.isfinite().all() for x in got)
        same = torch.ones(T, dtype=torch.bool, device=DEV)
        same[rows] = False
        assert torch.equal(got[0][:, same], want[:, same])
        if bad < 2:
            with pytest.raises(RuntimeError, match="outside its tree level"):
                ops.check_status()
    ops.check_status()


def _compare_with_generic(dt, D, CR, G, scales, tol_out, tol_grad):
    """Outputs and gradients of inputs times `scales` (q, k, v, dO) against the fp32-arithmetic kernels on the same saved state."""
    import htree_b200 as ht
    q, k, v, dO = (x * s for x, s in zip(_inputs(dt, 1, 1500, 2, G, D), scales))
    out, ctx = ht.htree_forward(q, k, v, CR, 64, 32, _save_for_backward=True)
    ref, rctx = ht.htree_forward(q, k, v, CR, 64, 32, _save_for_backward=True, _force_generic=True)
    same = torch.stack([(ctx["per_layer_parents"][l] == rctx["per_layer_parents"][l]).all(-1) for l in range(ctx["num_layers"])]).all(0)
    rows = same.repeat_interleave(G, -1)
    assert same.float().mean().item() >= 0.98
    rel = lambda a, b: ((a.double() - b.double()).norm() / b.double().norm()).item()
    assert rel(out[rows], ref[rows]) < tol_out
    for name, a, b in zip(("dq", "dk", "dv"), ht.htree_backward(dO, q, out, ctx), ht.htree_backward(dO, q, out, ctx, _force_generic=True)):
        assert rel(a, b) < tol_grad, (name, scales)


@pytest.mark.parametrize("dt,D,CR,G", [(FP, 128, 16, 8), (FP, 128, 8, 16), (FP, 64, 16, 4), (FP, 64, 8, 12), (FP, 32, 16, 4), (BF, 32, 16, 9),
                                       (BF, 32, 8, 4), (HF, 32, 8, 16)])
def test_range_of_split_half(dt, D, CR, G):
    """Half pairs carry fp32 values over a wider range than half's: a mean-reduced loss (dO of 1e-8), small and large values, small
    queries against large keys.  The tolerances are those of inputs near 1."""
    scales = [(1, 1, 1, 1), (1, 1, 3e-3, 3e-3)]
    if dt != HF:
        scales += [(1, 1, 1, 1e-8), (1, 1, 1, 1e6), (1, 1, 1e-6, 1), (1, 1, 1e6, 1), (1, 1, 1e4, 1e-6)]
        if D != 64:      # the selection of 64-wide heads reads the keys as they are
            scales += [(1e-5, 1e5, 1, 1), (1e5, 1e-5, 1, 1)]
    for s in scales:
        _compare_with_generic(dt, D, CR, G, s, 1e-5 if dt == FP else 4e-3, 1e-5)


@pytest.mark.parametrize("D,CR,G", [(128, 16, 8), (64, 8, 4), (32, 8, 9)])
def test_range_within_a_call(D, CR, G):
    """Groups, heads and blocks of very different magnitude in one call: each group and each block has its own scale, so a small
    gradient or value is as exact as it would be alone."""
    import htree_b200 as ht
    q, k, v, dO = _inputs(FP, 1, 1500, 2, G, D)
    dO[:, ::2] *= 1e-9                       # every other query: visits of both kinds share a parent
    v[:, 700:, 1] *= 1e-7
    q[:, 1::3] *= 1e-3
    out, ctx = ht.htree_forward(q, k, v, CR, 64, 32, _save_for_backward=True)
    ours, gen = ht.htree_backward(dO, q, out, ctx), ht.htree_backward(dO, q, out, ctx, _force_generic=True)
    for part in (slice(0, None, 2), slice(1, None, 2)):
        assert _rel(ours[0][:, part], gen[0][:, part]) < 1e-5
    for a, b in zip(ours[1:], gen[1:]):
        assert _rel(a[:, :, 0], b[:, :, 0]) < 1e-5 and _rel(a[:, :, 1], b[:, :, 1]) < 1e-5


@pytest.mark.parametrize("dt,D,CR,G", [(BF, 128, 16, 16), (BF, 128, 8, 5), (BF, 64, 16, 9), (BF, 64, 8, 8), (HF, 128, 16, 8), (HF, 64, 8, 16)])
def test_range_of_16_bit_gradients(dt, D, CR, G):
    """dS of the 16-bit kernels is a half: gradients keep their digits whatever the loss is divided by and however large the values."""
    scales = [(1, 1, 1, 1), (1, 1, 3e-3, 3e-3)]
    if dt == BF:
        scales += [(1, 1, 1, 1e-8), (1, 1, 1, 1e6), (1, 1, 1e-6, 1), (1, 1, 1e6, 1), (1, 1, 1e4, 1e-6)]
    for s in scales:
        _compare_with_generic(dt, D, CR, G, s, 4e-3, 3e-3)


@pytest.mark.parametrize("dt,D,T", [(BF, 128, 1), (BF, 64, 333), (HF, 128, 5000)])
def test_gradient_range_ignores_what_is_not_finite(dt, D, T):
    """The bound on dS is taken over finite rows: an infinite output gradient spoils its own head's gradient only."""
    import htree_b200 as ht
    q, k, v, dO = _inputs(dt, 1, T, 2, 4, D)
    out, ctx = ht.htree_forward(q, k, v, 16, 64, 32, _save_for_backward=True)
    want = ht.htree_backward(dO, q, out, ctx)[0]
    dO[:, -1, 0, 3] = float("inf")
    got = ht.htree_backward(dO, q, out, ctx)[0]
    if T > 1:
        # the other rows have the same bound, or half of it: dS rounds differently where it is subnormal (2^-25 of the bound)
        assert _rel(got[:, :-1], want[:, :-1]) < 1e-4
    assert got[:, -1, 4:].isfinite().all()


@pytest.mark.parametrize("dt,D,G,T,TK,MTN,Hkv,clustered", [
    (HF, 32, 4, 3001, 512, 8192, 4, False),      # every query reads everything there is: lists alike
    (FP, 32, 1, 5003, 512, 512, 2, False), (HF, 32, 2, 3001, 64, 512, 4, True), (BF, 32, 3, 2399, 64, 64, 4, False),
    (BF, 64, 4, 4001, 64, 256, 2, True), (HF, 64, 1, 3001, 64, 64, 4, False), (FP, 64, 3, 2048, 32, 64, 4, True), (FP, 64, 4, 2049, 32, 64, 4, False),
    (BF, 128, 4, 2047, 64, 128, 4, True), (HF, 128, 2, 4001, 128, 128, 4, False), (FP, 128, 4, 2049, 64, 64, 4, False)])
def test_queries_that_share_a_warp(dt, D, G, T, TK, MTN, Hkv, clustered):
    """Up to four queries of small groups walk the union of their lists in one warp.  Windows of too few queries for that take a warp
    each: their rows, and dq, are the same bits.  (Odd lengths: the last warp has fewer queries.)"""
    import htree_b200 as ht
    from htree_b200 import ops
    q, k, v, dO = _inputs(dt, 1, T, Hkv, G, D, clustered)
    dO = dO * (torch.rand(1, T, 1, 1, device=DEV) * 8 - 4).exp2().to(dt)       # neighbours of different size
    out, ctx = ht.htree_forward(q, k, v, 16, MTN, TK, _save_for_backward=True)
    ours, want = ht.htree_backward(dO, q, out, ctx), ht.htree_backward(dO, q, out, ctx, _force_generic=True)
    step, acc, outs, dqs = 1001 // Hkv, {}, [], []
    cuts = list(range(0, T, step)) + [T]
    for a, b in zip(cuts, cuts[1:]):
        qw = q[:, a:b].contiguous()
        o, c = ht.htree_forward(qw, k, v, 16, MTN, TK, _save_for_backward=True, _q_offset=a)
        r = ht.htree_backward(dO[:, a:b].contiguous(), qw, o, c, _window=dict(t0=a, first=a == 0, last=b == T, acc=acc))
        outs.append(o); dqs.append(r[0])
    assert torch.equal(torch.cat(outs, 1), out), "a row depends on the queries beside it"
    assert torch.equal(torch.cat(dqs, 1), ours[0]), "dq depends on the queries beside it"
    # sums in another order: 1e-6 relative; 16-bit dV takes P and dS takes dP in 16 bits, alike on both sides
    assert _rel(r[1], ours[1]) < 1e-5 and _rel(r[2], ours[2]) < 1e-5
    exact = dt == FP or D == 32
    if not clustered:      # (clustered scores reach 70: the half-precision operands of a score move its probability by a percent)
        for a, b in zip(ours, want):
            assert _rel(a, b) < (2e-5 if exact else 3e-3)
    torch.cuda.synchronize()
    ops.check_status()


@pytest.mark.parametrize("dt,D,G,T,TK,MTN,Hkv,CR,clustered", [
    (FP, 128, 8, 4096, 32, 256, 2, 16, False), (FP, 128, 16, 2100, 16, 256, 2, 16, True),   # tiles of 128 nodes: two, and one and a bit
    (FP, 128, 3, 3000, 128, 1024, 2, 16, False), (HF, 32, 4, 12000, 512, 8192, 4, 16, False),   # 750 nodes; a maximum and a sum per node
    (HF, 32, 8, 5000, 64, 512, 4, 8, True), (BF, 32, 12, 9001, 32, 128, 2, 8, False), (FP, 32, 1, 20000, 16, 64, 2, 16, False)])   # levels below
def test_top_level_in_fp32_arithmetic(dt, D, G, T, TK, MTN, Hkv, CR, clustered):
    """The dense product of the top level keeps exactly the nodes that one block per query keeps."""
    import htree_b200 as ht
    from htree_b200 import ops
    q, k, v, _ = _inputs(dt, 1, T, Hkv, G, D, clustered)
    lists = [ht.htree_forward(q, k, v, CR, MTN, TK, _save_for_backward=True, _force_generic=generic)[1]["per_layer_parents"] for generic in (False, True)]
    for l in lists[0]:
        assert torch.equal(lists[0][l], lists[1][l]), f"level {l}"
    torch.cuda.synchronize()
    ops.check_status()


@pytest.mark.parametrize("dt,D,G,T,TK,MTN,CR", [(FP, 128, 8, 2100, 16, 256, 16), (HF, 32, 4, 5000, 64, 512, 8), (FP, 32, 16, 4097, 32, 300, 16)])
def test_top_level_of_windows_and_rebuilt_lists(dt, D, G, T, TK, MTN, CR):
    """A window selects with the dense product from 592 groups on and with a block per query below, and a backward without saved lists
    rebuilds them with the latter: the same nodes throughout, for every batch row."""
    import htree_b200 as ht
    from htree_b200 import ops
    q, k, v, dO = _inputs(dt, 2, T, 2, G, D)
    out, ctx = ht.htree_forward(q, k, v, CR, MTN, TK, _save_for_backward=True)
    lists = ctx["per_layer_parents"]
    for w in (147, 148, 700):
        for t0 in (T - w, T // 2 + 1):
            _, c = ht.htree_forward(q[:, t0:t0 + w].contiguous(), k, v, CR, MTN, TK, _save_for_backward=True, _q_offset=t0)
            for l in lists:
                assert torch.equal(c["per_layer_parents"][l], lists[l][:, t0:t0 + w]), (w, t0, l)
    want = ht.htree_backward(dO, q, out, ctx)
    lists = {l: x.clone() for l, x in lists.items()}
    ctx["per_layer_parents"] = None
    rebuilt = ops.recompute_parents(q, ctx["layers_k"], ctx["layers_v"], ctx["cos_cache"], ctx["sin_cache"], CR, TK, MTN, ctx["scale"],
                                    layers_v_blk=ctx["layers_v_blk"], rope_base=ctx["rope_base"])
    for l in lists:
        assert torch.equal(rebuilt[l], lists[l]), l
    assert torch.equal(ht.htree_backward(dO, q, out, ctx)[0], want[0])
    torch.cuda.synchronize()
    ops.check_status()


@pytest.mark.parametrize("dt,D,G,T,TK,MTN,Hkv", [
    (HF, 32, 4, 1601, 64, 128, 4), (FP, 64, 3, 1600, 64, 128, 4), (BF, 128, 4, 1600, 64, 1024, 2),       # two queries a warp
    (BF, 64, 1, 1601, 64, 128, 4), (FP, 128, 2, 1603, 64, 128, 4)])                                      # four
@pytest.mark.parametrize("compact", [False, True])
def test_malformed_parent_lists_of_queries_that_share_a_warp(dt, D, G, T, TK, MTN, Hkv, compact, monkeypatch):
    """The union of lists that do not ascend has no more steps than the level has parents (101, where 64 entries of one parent and a
    neighbour's list would make 127), reports them, and leaves the other queries' gradients as they are."""
    import htree_b200 as ht
    from htree_b200 import ops
    if compact:
        monkeypatch.setattr(ops, "SELECTION_STORAGE", "uint16")
    q, k, v, dO = _inputs(dt, 1, T, Hkv, G, D)
    out, ctx = ht.htree_forward(q, k, v, 16, MTN, TK, _save_for_backward=True)
    want = ht.htree_backward(dO, q, out, ctx)
    lists = {l: x.clone() for l, x in ctx["per_layer_parents"].items()}
    rows = torch.arange(T // 2 | 1, T, 2, device=DEV)        # every other query of the later half: each warp has one as it should be
    same = torch.ones(T, dtype=torch.bool, device=DEV)
    same[rows] = False

    def one_parent(x): x[:, rows] = 3
    def descending(x): x[:, rows] = x[:, rows].flip(-1)
    def holes(x): x[:, rows, :, 1::2] = -1
    def first_missing(x): x[:, rows, :, 0] = -1
    def past_the_end(x): x[:, rows, :, 5] = -2 if compact else 1 << 30
    def twice(x): x[:, rows, :, 7] = x[:, rows, :, 6]
    for hurt in (one_parent, descending, holes, first_missing, past_the_end, twice):
        for levels in ([0], list(range(ctx["num_layers"]))):
            bad = {l: x.clone() for l, x in lists.items()}
            for l in levels:
                hurt(bad[l])
            ctx["per_layer_parents"] = bad
            got = ht.htree_backward(dO, q, out, ctx)
            torch.cuda.synchronize()
            assert all(x.isfinite().all() for x in got), hurt.__name__
            assert torch.equal(got[0][:, same], want[0][:, same]), hurt.__name__
            with pytest.raises(RuntimeError, match="outside its tree level"):
                ops.check_status()
    ctx["per_layer_parents"] = {l: x.clone() for l, x in lists.items()}
    for l in range(ctx["num_layers"]):
        ctx["per_layer_parents"][l][:, rows] = -1                # no parents at all: nothing to report
    got = ht.htree_backward(dO, q, out, ctx)
    assert torch.equal(got[0][:, same], want[0][:, same]) and not got[0][:, rows].any()
    ops.check_status()


@pytest.mark.parametrize("dt,D,G,T,TK,MTN,Hkv,CR", [
    (BF, 32, 4, 1600, 512, 8192, 4, 16), (BF, 32, 4, 1601, 512, 8192, 4, 16),       # two queries a warp; the last one beside the one before, or alone
    (FP, 32, 1, 1600, 512, 512, 4, 16), (BF, 32, 2, 1603, 64, 512, 4, 16),          # four
    (FP, 64, 4, 1600, 64, 64, 2, 16), (FP, 128, 3, 1602, 64, 64, 4, 16), (FP, 64, 4, 1500, 64, 64, 2, 8)])      # (eight children: one)
@pytest.mark.parametrize("of_dO,of_q", [(2.0 ** -4, 1), (2.0 ** -12, 1), (2.0 ** -24, 2.0 ** -8), (1, 2.0 ** -20), (1e-9, 1), (0, 1)])
def test_small_neighbours_keep_their_digits(dt, D, G, T, TK, MTN, Hkv, CR, of_dO, of_q):
    """The newest key is read by the newest query alone, whose visit shares its products with those of queries 1 / of_dO times as
    large: the key's gradients are as exact as if all were alike."""
    import htree_b200 as ht
    q, k, v, dO = _inputs(dt, 1, T, Hkv, G, D)
    dO[:, -1] *= of_dO
    q[:, -1] *= of_q
    out, ctx = ht.htree_forward(q, k, v, CR, MTN, TK, _save_for_backward=True)
    ours, want = ht.htree_backward(dO, q, out, ctx), ht.htree_backward(dO, q, out, ctx, _force_generic=True)
    for name, a, b in zip(("dq", "dk", "dv"), ours, want):          # (one row's dq is 1.3e-5 off at every scale)
        assert _rel(a[:, -1], b[:, -1]) < 2e-5 and _rel(a[:, :-1], b[:, :-1]) < 2e-5, name


# (Values of split halves and bf16 queries are clamped to half's range where they are read.)
@pytest.mark.parametrize("dt,D,G,T,TK,MTN,Hkv,what", [c + (w,) for c in (
    (BF, 64, 4, 2403, 64, 256, 2), (HF, 64, 1, 2401, 64, 64, 2), (BF, 128, 4, 2047, 64, 128, 2), (HF, 128, 2, 2401, 64, 128, 2),
    (HF, 32, 4, 2401, 64, 512, 2), (FP, 64, 2, 2402, 64, 64, 2), (FP, 128, 4, 2049, 64, 64, 2), (BF, 64, 4, 2403, 256, 4096, 2))
    for w in ("v", "q", "dO") if not (w == "v" and (c[0] == FP or c[1] == 32) or w == "q" and c[0] == BF)])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_what_is_not_finite_stays_with_the_queries_that_read_it(dt, D, G, T, TK, MTN, Hkv, what, bad):
    """Queries from position 1 on, so that some warps have queries on both sides of the start of a block: an infinite value there does not
    reach the query before it, nor that query's infinite q or dO the gradients of the block.  (NaN likewise.)"""
    import htree_b200 as ht
    from htree_b200 import ops
    q, k, v, dO = _inputs(dt, 1, T, Hkv, G, D)
    first = 1536                                 # (a block starts here on the level above too)
    if what == "v":
        v[:, first + 3, 0, 3] = bad
    else:
        (q if what == "q" else dO)[:, first - 1, G - 1, 5] = bad        # (of KV head 0)

    def windows(cuts):
        acc, outs, dqs = {}, [], []
        for a, b in zip(cuts, cuts[1:]):
            qw = q[:, a:b].contiguous()
            o, c = ht.htree_forward(qw, k, v, 16, MTN, TK, _save_for_backward=True, _q_offset=a)
            r = ht.htree_backward(dO[:, a:b].contiguous(), qw, o, c, _window=dict(t0=a, first=a == 1, last=b == T, acc=acc))
            outs.append(o); dqs.append(r[0])
        return torch.cat(outs, 1), torch.cat(dqs, 1), r[1], r[2]

    ours, want = windows([1, T - 1, T]), windows(list(range(1, T, 501)) + [T])       # (1002 groups and fewer: a warp each)
    assert not all(x.isfinite().all() for x in want)
    early, late = slice(0, first - 2), slice(first, None)
    assert all(x[:, early].isfinite().all() for x in want[:2])
    if what != "v":
        assert all(x[:, late].isfinite().all() for x in want[2:])
    for name, a, b in zip(("out", "dq", "dk", "dv"), ours, want):
        fine = b.isfinite()
        assert torch.equal(a.isfinite(), fine), name
        if name in ("out", "dq"):
            fine[:, first - 2] = False                  # (the query itself: its dS is scaled by the call's largest dO, which it is left out of)
            assert torch.equal(a[fine], b[fine]), name
        else:
            assert not fine.any() or _rel(a[fine], b[fine]) < 1e-5, name
    torch.cuda.synchronize()
    ops.check_status()


@pytest.mark.parametrize("D,G,Hkv,CR", [(32, 8, 2, 16), (32, 4, 4, 16), (64, 2, 4, 16), (128, 8, 2, 8), (64, 16, 2, 8)])
@pytest.mark.parametrize("size", [1e6, 1e20])
def test_no_gradient_beside_large_values(D, G, Hkv, CR, size):
    """Queries without an output gradient have dq = 0 and add nothing, however large the values (the scale of their dS, from a bound of
    zero, was 2^124)."""
    import htree_b200 as ht
    q, k, v, dO = _inputs(FP, 1, 2000, Hkv, G, D)
    v *= size
    dO /= size
    dO[:, 1000:1101] = 0
    out, ctx = ht.htree_forward(q, k, v, CR, 64, 32, _save_for_backward=True)
    ours, want = ht.htree_backward(dO, q, out, ctx), ht.htree_backward(dO, q, out, ctx, _force_generic=True)
    assert not ours[0][:, 1000:1101].any()
    for name, a, b in zip(("dq", "dk", "dv"), ours, want):
        assert ((a.double() - b.double()).norm() / b.double().norm()).item() < 1e-5, name


@pytest.mark.parametrize("dt,D,G,T,TK,MTN,Hkv", [(FP, 64, 2, 2402, 64, 64, 2), (FP, 128, 4, 2049, 64, 64, 4), (FP, 32, 4, 2403, 64, 512, 2)])
@pytest.mark.parametrize("what", ["v", "k"])
def test_what_overflows_stays_with_the_queries_that_read_it(dt, D, G, T, TK, MTN, Hkv, what):
    """Values and keys near the end of fp32's range, as above: their factors, times another query's, are infinite, and so are the sums of
    the queries that read them."""
    import htree_b200 as ht
    q, k, v, dO = _inputs(dt, 1, T, Hkv, G, D)
    first = 1536
    if what == "v":
        v[:, first + 3, 0, 3] = 3e38
    else:
        k[:, first + 3, 0, 3] = 3e38
        dO *= 1e8

    def windows(cuts):
        acc, outs, dqs = {}, [], []
        for a, b in zip(cuts, cuts[1:]):
            qw = q[:, a:b].contiguous()
            o, c = ht.htree_forward(qw, k, v, 16, MTN, TK, _save_for_backward=True, _q_offset=a)
            r = ht.htree_backward(dO[:, a:b].contiguous(), qw, o, c, _window=dict(t0=a, first=a == 1, last=b == T, acc=acc))
            outs.append(o); dqs.append(r[0])
        return torch.cat(outs, 1), torch.cat(dqs, 1), r[1], r[2]

    ours, want = windows([1, T - 1, T]), windows(list(range(1, T, 501)) + [T])       # (1002 groups and fewer: a warp each)
    early = slice(0, first - 1)                                                       # (row 0 is position 1)
    for name, a, b in zip(("out", "dq", "dk", "dv"), ours, want):
        fine = b.isfinite()
        assert torch.equal(a.isfinite(), fine), name
        if name in ("out", "dq"):
            assert fine[:, early].all() and torch.equal(a[:, early], b[:, early]), name
        a, b = a[fine].double(), b[fine].double()
        assert ((a - b).norm() / b.norm()).item() < 1e-5, name
    torch.cuda.synchronize()


@pytest.mark.parametrize("dt,D,G,T,TK,MTN,Hkv,CR", [(FP, 128, 8, 4096, 32, 256, 2, 16), (HF, 32, 4, 12000, 512, 8192, 2, 16), (BF, 32, 8, 5000, 64, 512, 2, 8)])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_top_level_with_what_is_not_finite(dt, D, G, T, TK, MTN, Hkv, CR, bad):
    """Lists of queries that see no infinite key are those of one block per query, whatever the queries and keys of their tile hold; the
    others name nodes that exist, ascending."""
    import htree_b200 as ht
    from htree_b200 import ops
    q, k, v, _ = _inputs(dt, 1, T, Hkv, G, D)
    q[:, 100::7, 1, 3] = bad
    k[:, T // 2, :, 5] = bad
    lists = []
    for generic in (False, True):
        _, ctx = ht.htree_forward(q, k, v, CR, MTN, TK, _save_for_backward=True, _force_generic=generic)
        lists.append(ctx["per_layer_parents"])
    L = ctx["num_layers"]
    seen = torch.arange(T, device=DEV) // CR ** (L - 1) >= T // 2 // CR ** (L - 1)        # (from the top level's node of that key on)
    own = torch.zeros(T, Hkv, dtype=torch.bool, device=DEV)
    own[100::7, 0] = True                                                                # (head 1 belongs to KV head 0)
    clean = ~(seen[:, None] | own)
    assert 0.2 < clean.float().mean().item() < 0.8
    n = T
    for l in range(L):
        ours, want = lists[0][l][0], lists[1][l][0]
        n = (n + CR - 1) // CR                                                           # the parents of level l
        assert torch.equal(ours[clean], want[clean]), f"level {l}"
        assert ours.min().item() >= -1 and ours.max().item() < n
        assert ((ours[..., 1:] > ours[..., :-1]) | (ours[..., 1:] == -1)).all()
    torch.cuda.synchronize()
    ops.check_status()
