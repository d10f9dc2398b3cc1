"""Each kernel alone against a plain float32/float64 reference of the same operation, at
sizes other than the engine's: widths that are no power of two, odd row counts, head
sizes in steps of 16, several page sizes. Inputs are built so that faults show: a far
key that dominates a softmax, a window's edge, values in unused pages that would
poison a result if read."""


import pytest
import torch

from kernel_refs import build_pages, ref_paged_attention
from plain.plain_qwen3 import plain_sample

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _k():
    from quantinfer_b200 import kernels
    return kernels


def _status():
    return torch.zeros(1, dtype=torch.int32, device=DEV)


def I(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


# ------------------------------------------------------------------ embedding, norms

@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("vocab, hidden", [(37, 20), (300, 168), (1000, 4096)])
def test_embedding(dtype, vocab, hidden):
    torch.manual_seed(0)
    table = torch.randn(vocab, hidden).to(dtype).to(DEV)
    ids = torch.randint(0, vocab, (13,), dtype=torch.int32)
    out = torch.empty(13, hidden, dtype=torch.float32, device=DEV)
    st = _status()
    _k().embedding(table, ids.to(DEV), out, st)
    assert torch.equal(out.cpu(), table.float().cpu()[ids.long()]) and st.item() == 0
    bad = ids.clone()
    bad[3] = vocab
    _k().embedding(table, bad.to(DEV), out, st)
    assert st.item() == _k().STATUS_BAD_TOKEN and float(out[3].abs().max()) == 0.0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows, hidden", [(1, 20), (7, 168), (5, 4096), (3, 1000)])
def test_add_rmsnorm(dtype, rows, hidden):
    torch.manual_seed(1)
    resid = torch.randn(rows, hidden)
    delta = torch.randn(rows, hidden).to(dtype)
    gain = 1 + 0.1 * torch.randn(hidden)
    eps = 3e-6
    x = resid.double() + delta.double()
    ref = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * gain.double()
    r = resid.to(DEV)
    out = torch.empty(rows, hidden, dtype=dtype, device=DEV)
    _k().add_rmsnorm(r, delta.to(DEV), gain.to(DEV), eps, out)
    tol = 1e-5 if dtype == torch.float32 else 2e-2
    assert float((out.double().cpu() - ref).abs().max()) < tol
    assert float((r.double().cpu() - x).abs().max()) < 1e-6           # the residual stream was updated
    # no delta, row gather, residual untouched
    r2 = resid.to(DEV)
    pick = I([rows - 1, 0])
    out2 = torch.empty(2, hidden, dtype=dtype, device=DEV)
    _k().add_rmsnorm(r2, None, gain.to(DEV), eps, out2, rows=pick)
    x2 = resid.double()[[rows - 1, 0]]
    ref2 = x2 * torch.rsqrt((x2 * x2).mean(-1, keepdim=True) + eps) * gain.double()
    assert float((out2.double().cpu() - ref2).abs().max()) < tol and torch.equal(r2.cpu(), resid)


@pytest.mark.parametrize("rows, hidden, splits", [
    (6, 264, 3),          # one CTA a row
    (8, 4096, 8),         # few rows of a wide model: a row over a cluster of four CTAs, all partial sums at once
    (64, 1024, 2),        # the most rows and the narrowest rows that take the clusters
    (3, 5120, 16),        # more partial sums than are requested at once
    (65, 4096, 4),        # one row too many for the clusters
    (1500, 2048, 2),      # more rows than CTAs that stay: each walks several rows
])
def test_add_rmsnorm_takes_split_partials(rows, hidden, splits):
    torch.manual_seed(2)
    resid, parts = torch.randn(rows, hidden), torch.randn(splits, rows, hidden)
    gain = 1 + 0.1 * torch.randn(hidden)
    x = resid.double() + parts.double().sum(0)
    ref = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6) * gain.double()
    out = torch.empty(rows, hidden, dtype=torch.bfloat16, device=DEV)
    r = resid.to(DEV)
    _k().add_rmsnorm(r, parts.to(DEV), gain.to(DEV), 1e-6, out)
    assert float((out.double().cpu() - ref).abs().max()) < 3e-2 and float((r.double().cpu() - x).abs().max()) < 1e-5
    # the same sums for picked rows only (what the head's norm does): the residual stays as it was
    r2 = resid.to(DEV)
    pick = [rows - 1, 0]
    out2 = torch.empty(2, hidden, dtype=torch.float32, device=DEV)
    _k().add_rmsnorm(r2, parts.to(DEV), gain.to(DEV), 1e-6, out2, rows=I(pick))
    assert float((out2.double().cpu() - ref[pick]).abs().max()) < 2e-5 and torch.equal(r2.cpu(), resid)


# ------------------------------------------------------------------ matrix products

@pytest.mark.parametrize("tx, tw, ty", [(torch.float32,) * 3, (torch.bfloat16,) * 3,
                                        (torch.bfloat16, torch.float32, torch.bfloat16),
                                        (torch.bfloat16, torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("M, N, K", [(1, 7, 5), (65, 130, 33), (200, 517, 168)])
def test_gemm_simt(tx, tw, ty, M, N, K):
    torch.manual_seed(3)
    x, w = torch.randn(M, K).to(tx), torch.randn(N, K).to(tw)
    out = torch.empty(M, N, dtype=ty, device=DEV)
    _k().gemm_simt(x.to(DEV), w.to(DEV), out)
    ref = x.double() @ w.double().t()
    tol = 1e-4 if ty == torch.float32 else 0.15
    assert float((out.double().cpu() - ref).abs().max()) < tol


@pytest.mark.parametrize("N, K", [(1, 4), (33, 68), (517, 168), (4096, 260), (6000, 96)])
@pytest.mark.parametrize("M", [1, 16, 17, 40, 65, 112, 113, 201, 300])
def test_gemm_f32_keeps_the_order_of_its_sums(M, N, K):
    """The copied-tile kernel (32-bit operands, rows of whole 16-byte pieces) against the element-wise one, which takes the
    same numbers when the weights come as bfloat16: bit for bit the same, over the edges of every tile."""
    torch.manual_seed(M + N)
    x, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV).to(torch.bfloat16)
    fast, plain_ = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    _k().gemm_simt(x, w.float(), fast)
    _k().gemm_simt(x, w, plain_)
    assert torch.equal(fast, plain_)
    # the error of k in order: at most K roundings of 2^-24 of the sum of magnitudes
    bound = K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    assert bool(((fast.double() - x.double() @ w.double().T).abs() <= bound).all())


def test_gemm_simt_reads_what_the_kernel_before_it_wrote():
    """Both operands may be another kernel's results: a chain of products whose second operand the launch before wrote, over buffers that
    hold other numbers before."""
    torch.manual_seed(2)
    k, n = _k(), 1024
    a = torch.randn(n, n, device=DEV) * n ** -0.5
    steps = [torch.randn(n, n, device=DEV) * n ** -0.5 for _ in range(2)]
    for small in (False, True):
        x = a[:24].contiguous() if small else a
        want, w = [], a
        for i in range(12):
            w = steps[i % 2].double() @ w.double().T
            want.append(x.double() @ w.T)
        got, bufs, w = [], [torch.full((n, n), 1e3, device=DEV) for _ in range(12)], a
        for i in range(12):
            k.gemm_simt(steps[i % 2], w, bufs[i])
            got.append(torch.full((x.shape[0], n), -1e3, device=DEV))
            k.gemm_simt(x, bufs[i], got[-1])
            w = bufs[i]
        # each product's error is at most K 2^-24 of the sum of magnitudes, which is about 32 times the result here; twelve in a row
        assert max(float((g.double() - r).norm() / r.norm()) for g, r in zip(got, want)) < 12 * 32 * n * 2.0 ** -24


@pytest.mark.parametrize("N, K", [(4096, 1024), (1028, 4096), (512, 8192), (70000, 64), (1024, 4160)])
def test_gemm_f32_on_tensor_cores(N, K):
    """Three bfloat16 parts an operand: no further from 64 bits than the chain of single FMAs, over the edges of the token tiles; a row is the
    same alone and among others."""
    torch.manual_seed(N)
    k = _k()
    w = torch.randn(N, K, device=DEV) * 0.02
    assert k.library().qi_gemm_f32_workspace(1, N, K) > 0
    full = torch.randn(300, K, device=DEV) * torch.logspace(-3, 3, 300, device=DEV)[:, None]
    whole = torch.empty(300, N, device=DEV)
    k.gemm_f32(full, w, whole)
    ref = full.double() @ w.double().T
    chain = torch.empty(300, N, device=DEV)
    k.gemm_simt(full, w, chain)
    off = lambda y: float(((y.double() - ref).norm(dim=1) / ref.norm(dim=1)).mean())  # noqa: E731
    assert off(whole) <= off(chain)
    for M in (1, 15, 16, 17, 127, 128, 129, 257):
        out = torch.empty(M, N, device=DEV)
        k.gemm_f32(full[300 - M:].contiguous(), w, out)
        assert torch.equal(out, whole[300 - M:])


@pytest.mark.parametrize("M", [1023, 1025, 2100])
def test_gemm_f32_on_tensor_cores_rows_in_passes(M):
    """More rows than go through the workspace at a time: every row is what it is alone, with K whole and in parts, and the workspace does not grow."""
    torch.manual_seed(M)
    k = _k()
    for N, K in ((70000, 64), (1028, 4096)):
        x, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV) * 0.02
        x[M - 1, 3] = float("inf")
        got = torch.empty(M, N, device=DEV)
        k.gemm_f32(x, w, got)
        for a, b in ((0, 128), (1000, M), (M - 1, M)):
            part = torch.empty(b - a, N, device=DEV)
            k.gemm_f32(x[a:b].contiguous(), w, part)
            assert torch.equal(part.nan_to_num(1e9), got[a:b].nan_to_num(1e9))
        assert k.library().qi_gemm_f32_workspace(M, N, K) <= k.library().qi_gemm_f32_workspace(1024, N, K)


def test_gemm_f32_on_tensor_cores_numbers_without_parts():
    """Infinities, NaN and numbers that round to infinity as a bfloat16: what the chain of FMAs makes of them, and no other row or column
    notices. Parts of K are added, so that finite results may differ in their last bits."""
    torch.manual_seed(7)
    k, N, K, M = _k(), 2048, 2048, 40
    x, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)
    clean = torch.empty(M, N, device=DEV)
    k.gemm_f32(x, w, clean)
    x[3, 5], x[4, 2000], x[17, 0] = float("inf"), float("nan"), 3.4e38
    w[9, 100], w[300, 7], w[301, 2047] = float("-inf"), float("nan"), -3.4e38
    x[20] = 0.0
    x[21, 100] = 0.0
    got, chain = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    k.gemm_f32(x, w, got)
    k.gemm_simt(x, w, chain)
    assert torch.equal(got.isnan(), chain.isnan()) and torch.equal(got.isinf(), chain.isinf())
    assert torch.equal(got[chain.isinf()], chain[chain.isinf()])
    fine = chain.isfinite()
    bound = K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)
    assert bool(((got.double() - chain.double()).abs()[fine] <= bound[fine]).all())
    rows, cols = [i for i in range(M) if i not in (3, 4, 17, 20, 21)], [i for i in range(N) if i not in (9, 300, 301)]
    assert torch.equal(got[rows][:, cols], clean[rows][:, cols])


@pytest.mark.parametrize("N, K", [(70000, 64), (2048, 2048)])      # K whole, and in parts
def test_gemm_f32_on_tensor_cores_far_from_one(N, K):
    """Finite operands whose products or sums leave the range of 32-bit numbers give what the chain of FMAs gives, bit for bit, and no
    other result notices; so do rows of x or w that hold nothing above 2^-86, whose parts would lose bits. K stays far below the
    range of tiny numbers beside larger ones: their lost bits are 2^-48 of the largest."""
    torch.manual_seed(11)
    k, M = _k(), 40
    x, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)
    assert k.library().qi_gemm_f32_workspace(M, N, K) > 0
    clean, got, chain = (torch.empty(M, N, device=DEV) for _ in range(3))
    k.gemm_f32(x, w, clean)
    # products far above the range, with remainders of both signs; near the largest number; infinite one way, then the other
    x[3, 5], w[9, 5] = 1.00390625e25, 1.00390625e25
    x[4, K - 1], w[10, K - 1] = 1.003e25, -1.0045e25
    x[5, 0], w[11, 0] = 1.8446743e19, 1.8446743e19
    x[6, 1], w[12, 1] = 1.30e19, 2.617e19
    x[7, 2], x[7, K - 2], w[13, 2], w[13, K - 2] = 1e30, -1e30, 1e30, 1e30
    x[8, 3], x[8, K - 3], w[14, 3], w[14, K - 3] = 1e30, -1e30, 1e8, 1e8        # 1e38 - 1e38
    # rows of tiny numbers; tiny ones beside others
    x[20] *= 2.0 ** -115
    x[21] *= 2.0 ** -100
    w[300] *= 2.0 ** -112
    w[301] *= 2.0 ** -130
    x[22, ::2] *= 2.0 ** -115
    w[302, 1::2] *= 2.0 ** -115
    k.gemm_f32(x, w, got)
    k.gemm_simt(x, w, chain)
    assert bool(chain[3, 9].isinf()) and bool(chain[5, 11].isfinite()) and bool(chain[8, 14].isfinite())
    out_of_range = ~chain.isfinite()
    assert torch.equal(got[out_of_range], chain[out_of_range]) and bool(got[~out_of_range].isfinite().all())
    assert torch.equal(got[20:22], chain[20:22]) and torch.equal(got[:, 300:302], chain[:, 300:302])
    # twice the chain's own bound: K roundings of 2^-24 of the sum of magnitudes
    bound = K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)
    assert bool(((got.double() - chain.double()).abs() <= bound)[~out_of_range].all())
    rows = [i for i in range(M) if i not in (3, 4, 5, 6, 7, 8, 20, 21, 22)]
    cols = [i for i in range(N) if i not in (9, 10, 11, 12, 13, 14, 300, 301, 302)]
    assert torch.equal(got[rows][:, cols], clean[rows][:, cols])


FORMS = {   # M, N, K, plan
    "weights on the rows": (33, 70000, 512, (1, 64, 1)), "tokens on the rows": (2300, 4096, 512, (0, 256, 1)),
    "tokens on pairs": (1100, 8192, 512, (2, 256, 1)), "three parts": (201, 4096, 1024, None),
    "groups": (1100, 4096, 512, None), "attention": (1400, 4, 128, None)}


@pytest.mark.parametrize("form", FORMS)
def test_a_launch_after_a_wait_that_ran_out_leaves(form):
    """With the bit of a wait that ran out in the status word a launch on the tensor cores leaves instead of computing (its blocks have
    several tiles, so that roles are at every place when they learn of it) and keeps the bit; cleared, it computes."""
    torch.manual_seed(3)
    k, st = _k(), _status()
    M, N, K, plan = FORMS[form]
    if form == "attention":
        nkv, ps, pages, first = 2, 64, -(-M // 64), list(range(0, M, k.QUERY_TILE))
        kp, vp = (torch.randn(pages, nkv, ps, K, device=DEV).bfloat16() for _ in range(2))
        q, got = torch.randn(M, N * K, device=DEV).bfloat16(), torch.empty(M, N * K, dtype=torch.bfloat16, device=DEV)

        def run():
            k.attention_prefill(q, got, kp, vp, I([list(range(pages))]), I([0, M]), I([0]), I([0] * len(first)), I(first), N, nkv, K, K ** -0.5, 0, st,
                                impl="tcgen05")

        keys, vals = (p.transpose(1, 2).reshape(-1, nkv, K)[:M].double().repeat_interleave(N // nkv, dim=1) for p in (kp, vp))
        s = torch.einsum("ihd,jhd->hij", q.view(M, N, K).double(), keys) * K ** -0.5
        s.masked_fill_(torch.ones(M, M, dtype=torch.bool, device=DEV).triu(1), float("-inf"))
        ref = torch.einsum("hij,jhd->ihd", torch.softmax(s, dim=2), vals).reshape(M, N * K)
    else:
        groups = [0, 300, 300, 701, M] if form == "groups" else [0, M]
        dtype = torch.float32 if form == "three parts" else torch.bfloat16
        x, w = torch.randn(M, K, device=DEV).to(dtype), torch.randn(len(groups) - 1, N, K, device=DEV).to(dtype)
        got = torch.empty(M, N, dtype=dtype, device=DEV)

        def run():
            if form == "three parts":
                k.gemm_f32(x, w[0], got, status=st)
            elif form == "groups":
                k.gemm_bf16_grouped(x, w, got, I(groups), st)
            else:
                k.gemm_bf16(x, w[0], got, plan=plan, status=st)

        ref = torch.cat([x[a:b].double() @ w[g].double().T for g, (a, b) in enumerate(zip(groups, groups[1:]))])
    st.fill_(k.STATUS_WAIT_TIMEOUT)
    run()
    assert st.item() == k.STATUS_WAIT_TIMEOUT
    st.zero_()
    run()
    # half a unit of 2^-8 of the largest value; the attention's weights are rounded to bfloat16 too
    assert st.item() == 0 and float((got.double() - ref).abs().max()) <= float(ref.abs().max()) * 2.0 ** -8


@pytest.mark.parametrize("rows, N, K", [
    ([1], 2, 8), ([32, 33, 0, 31], 256, 64), ([190, 0, 256, 257, 5], 384, 136), ([513, 1, 700], 130, 1032), ([0, 0, 0, 2305], 254, 72),
    ([7] * 150, 512, 264), ([0, 0], 64, 64),
])
@pytest.mark.parametrize("epilogue", [None, "silu_mul", "glu_clamped"])
def test_gemm_bf16_grouped(rows, N, K, epilogue):
    """Every group's rows with its own weights, over the edges of the tiles (32, 256 rows; 256 weight rows), empty groups, more tiles than
    pairs; rows of no group stay as they were."""
    torch.manual_seed(N)
    E, n, spare = len(rows), sum(rows), 3
    x, w = torch.randn(n + spare, K, device=DEV).to(torch.bfloat16), (torch.randn(E, N, K, device=DEV) * K ** -0.5).to(torch.bfloat16)
    off = [0]
    for r in rows:
        off.append(off[-1] + r)
    out = torch.full((n + spare, N // 2 if epilogue else N), 77.0, device=DEV, dtype=torch.bfloat16)
    status = I([0])
    _k().gemm_bf16_grouped(x, w, out, I(off), status, epilogue=epilogue, glu=(1.0, 1.7) if epilogue == "glu_clamped" else None)
    assert int(status) == 0 and bool((out[n:] == 77.0).all())
    for e in range(E):
        ref = x[off[e]:off[e + 1]].double() @ w[e].double().T
        if epilogue:
            g, u = ref[:, 0::2], ref[:, 1::2]
            if epilogue == "silu_mul":
                ref = g * torch.sigmoid(g) * u
            else:
                g, u = g.clamp(max=1.0), u.clamp(-1.0, 1.0)
                ref = g * torch.sigmoid(1.7 * g) * (u + 1.0)
        # rounding to bfloat16 (2^-9) beside the 32-bit sums of products of order one
        assert bool(((out[off[e]:off[e + 1]].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("d, dv, window, keep", [(8, 8, 0, 0), (16, 16, 0, 0), (128, 128, 0, 0), (64, 40, 9, 2), (256, 200, 33, 0)])
def test_attention_generic_by_pieces_and_by_elements(dtype, d, dv, window, keep):
    """Keys read in 16-byte pieces and one by one (pages that start off a 16-byte boundary): bit for bit the same, on a page table with
    a page that is not there, too."""
    torch.manual_seed(d)
    nq, nkv, page, pages, n = 4, 2, 16, 9, 130
    kp, vp = torch.randn(pages, nkv, page, d, device=DEV).to(dtype), torch.randn(pages, nkv, page, dv, device=DEV).to(dtype)
    q = torch.randn(n, nq * d, device=DEV).to(dtype)
    shifted = torch.empty(kp.numel() + 1, dtype=dtype, device=DEV)[1:].view(kp.shape)
    shifted.copy_(kp)
    table, pos, req = I([[4, 0, 7, 2, 8, 1, 3, 5, 6], [1, 2, -1, 3, 4, 5, 6, 7, 8]]), I(list(range(n))), I([i % 2 for i in range(n)])
    got = []
    for keys in (kp, shifted):
        out, status = torch.empty(n, nq * dv, dtype=dtype, device=DEV), I([0])
        _k().attention_generic(q, out, keys, vp, table, pos, req, nq, nkv, d, d ** -0.5, window, status, keep_first=keep)
        got.append((out, int(status)))
    assert torch.equal(got[0][0], got[1][0]) and got[0][1] == got[1][1] == 2
    # request 0, whose pages are all there, against 64 bits
    keys = kp[table[0].long()].transpose(1, 2).reshape(pages * page, nkv, d).double()
    vals = vp[table[0].long()].transpose(1, 2).reshape(pages * page, nkv, dv).double()
    j, t = torch.arange(pages * page, device=DEV), torch.arange(0, n, 2, device=DEV)
    seen = (j[None] <= t[:, None]) & ((j[None] > t[:, None] - window) | (j[None] < keep) if window else torch.ones_like(j[None], dtype=torch.bool))
    for h in range(nq):
        s = (q.view(n, nq, d)[t, h].double() @ keys[:, h // 2].T) * d ** -0.5
        ref = torch.softmax(s.masked_fill(~seen, float("-inf")), dim=1) @ vals[:, h // 2]
        # 32-bit sums of at most 256 terms (1e-5 of values of order 4); a result in bfloat16 is rounded by 2^-9
        assert float((got[0][0].view(n, nq, dv)[t, h].double() - ref).abs().max()) < (2e-5 if dtype == torch.float32 else 2e-5 + 4 * 2.0 ** -8)


@pytest.mark.parametrize("M, N, K, plan", [
    (128, 128, 64, (False, 128, 1)), (100, 72, 136, (False, 64, 1)), (300, 520, 264, None),
    (4, 128, 64, (True, 16, 1)), (1, 384, 96, None), (33, 517, 168, (True, 64, 2)),
    (64, 1000, 2048, None), (200, 300, 4096, None), (700, 328, 168, (False, 256, 1)), (17, 264, 1032, (True, 32, 4)),
    # pairs of CTAs on tiles of 256 x 256: one tile, ragged edges in both directions, many k blocks, more tiles than pairs
    (256, 256, 64, (2, 256, 1)), (300, 400, 136, (2, 256, 1)), (129, 130, 1032, (2, 256, 1)), (2560, 2304, 320, (2, 256, 1)),
    (512, 300, 2048, (2, 256, 3)), (700, 1100, 1600, (2, 256, 2)),      # the same with K split: partial sums, then added
    # plans of width 0, whose width is not read (the same kernel of pairs): one tile, ragged edges, K split, more tiles than pairs
    (1, 256, 64, (2, 0, 1)), (33, 130, 136, (2, 0, 1)), (516, 520, 1032, (2, 0, 1)), (257, 2304, 320, (2, 0, 1)),
    (2305, 1026, 192, (2, 0, 1)), (65, 300, 2048, (2, 0, 3)), (700, 1100, 1600, (2, 0, 2)), (129, 9000, 520, (2, 0, 3)),
])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_tcgen05(M, N, K, plan, out_dtype):
    torch.manual_seed(4)
    x, w = (torch.randn(M, K) * 0.5).bfloat16(), (torch.randn(N, K) * 0.5).bfloat16()
    out = torch.full((M, N), 7.0, dtype=out_dtype, device=DEV)
    st = _status()
    _k().gemm_bf16(x.to(DEV), w.to(DEV), out, plan=plan, status=st)
    ref = x.double() @ w.double().t()
    err = float((out.double().cpu() - ref).abs().max())
    scale = float(ref.abs().max())
    assert st.item() == 0
    assert err < (2e-4 if out_dtype == torch.float32 else scale * 2 ** -7), (err, scale)


@pytest.mark.parametrize("M, N, K", [(5, 256, 136), (130, 328, 264), (64, 4096, 512)])
def test_gemm_tcgen05_silu_epilogue_and_partials(M, N, K):
    torch.manual_seed(5)
    x, w = (torch.randn(M, K) * 0.3).bfloat16(), (torch.randn(N, K) * 0.3).bfloat16()
    act = torch.empty(M, N // 2, dtype=torch.bfloat16, device=DEV)
    _k().gemm_bf16(x.to(DEV), w.to(DEV), act, epilogue="silu_mul")
    y = x.double() @ w.double().t()
    g, u = y[:, 0::2], y[:, 1::2]
    ref = g / (1 + torch.exp(-g)) * u
    assert float((act.double().cpu() - ref).abs().max()) < max(0.05, float(ref.abs().max()) * 2 ** -7)
    parts = _k().gemm_bf16(x.to(DEV), w.to(DEV), None, plan=(True if M <= 256 else False, 16 if M <= 16 else 256 if M > 64 else 64, 2),
                           keep_partials=True)
    assert parts.shape == (2, M, N) and float((parts.double().sum(0).cpu() - y).abs().max()) < 2e-4
    parts = _k().gemm_bf16(x.to(DEV), w.to(DEV), None, plan=(2, 256, 2), keep_partials=True)     # on pairs of CTAs
    assert parts.shape == (2, M, N) and float((parts.double().sum(0).cpu() - y).abs().max()) < 2e-4
    # the same activation from the kernel that runs on pairs of CTAs
    act2 = torch.empty_like(act)
    _k().gemm_bf16(x.to(DEV), w.to(DEV), act2, plan=(2, 256, 1), epilogue="silu_mul")
    assert float((act2.double().cpu() - ref).abs().max()) < max(0.05, float(ref.abs().max()) * 2 ** -7)


def test_gemm_plan_takes_cta_pairs_for_many_tokens():
    k = _k()
    assert k.gemm_bf16_plan(2048, 4096, 4096)[0] == 2 and k.gemm_bf16_plan(2048, 24576, 4096, allow_split=False)[0] == 2
    assert k.gemm_bf16_plan(8, 4096, 4096)[0] == 1 and k.gemm_bf16_plan(64, 24576, 4096)[0] == 1


# ------------------------------------------------------------------ q/k norm, rotation, cache write

@pytest.mark.parametrize("M, K, nq, nkv, ps, norm, rope, write", [
    (300, 64, 2, 1, 16, True, True, True),      # 4 heads: two tiles of 256 columns; a ragged last row tile
    (257, 136, 3, 1, 8, True, True, True),      # 5 heads: the last tile is half empty; K no multiple of 64
    (513, 256, 1, 1, 64, False, True, True),    # 3 heads: one tile of 256 and a half; no norm
    (384, 72, 1, 2, 32, True, False, True),     # no rotation
    (260, 64, 2, 1, 16, True, True, False),     # reads another layer's cache: queries only
    (1300, 64, 12, 4, 16, True, True, True),    # 20 heads, many tokens: the kernel on pairs of CTAs
    (1100, 136, 9, 3, 64, True, True, True),    # 15 heads: the pair's last tile holds one head only
])
def test_gemm_qkv_rope(M, K, nq, nkv, ps, norm, rope, write):
    """The q/k/v projection with norm, rotation and cache write in its epilogue, against a 64-bit
    product followed by the formulas; heads that straddle tile borders, rows past the last token."""
    torch.manual_seed(M + K)
    d, eps, theta, max_pos = 128, 1e-5, 1e4, 1400
    k = _k()
    assert k.gemm_qkv_rope_supported(M, K, d, d if rope else 0, torch.bfloat16, torch.bfloat16)
    assert not k.gemm_qkv_rope_supported(200, K, d, d, torch.bfloat16, torch.bfloat16)
    assert not k.gemm_qkv_rope_supported(M, K, 64, 64, torch.bfloat16, torch.bfloat16)
    x = torch.randn(M, K).bfloat16()
    w = (torch.randn((nq + 2 * nkv) * d, K) / K ** 0.5).bfloat16()
    qg, kg = (1 + 0.1 * torch.randn(d), 1 + 0.1 * torch.randn(d)) if norm else (None, None)
    inv_freq = torch.pow(torch.tensor(theta), -(2.0 * torch.arange(d // 2)) / d)
    cos, sin = k.rope_table(inv_freq.to(DEV), max_pos) if rope else (None, None)
    ang = torch.arange(max_pos, dtype=torch.float64)[:, None] * inv_freq.double()[None, :]
    # two requests: the first holds 40 earlier positions, the second starts at 0
    n0 = M // 3
    positions = list(range(40, 40 + n0)) + list(range(0, M - n0))
    token_req = [0] * n0 + [1] * (M - n0)
    max_blocks = -(-max_pos // ps)
    num_pages = 2 * max_blocks + 3
    perm = torch.randperm(num_pages).tolist()
    table = torch.tensor([[perm.pop() for _ in range(max_blocks)] for _ in range(2)], dtype=torch.int32)
    kp = torch.zeros(num_pages, nkv, ps, d, dtype=torch.bfloat16, device=DEV)
    vp = torch.zeros_like(kp)
    q_out = torch.empty(M, nq * d, dtype=torch.bfloat16, device=DEV)
    st = _status()
    k.gemm_qkv_rope(x.to(DEV), w.to(DEV), q_out, qg.to(DEV) if norm else None, kg.to(DEV) if norm else None, eps, cos, sin,
                    I(positions), I(token_req), table.to(DEV), ps, kp if write else None, vp if write else None, nq, nkv, st)
    assert st.item() == 0
    y = (x.double() @ w.double().T).reshape(M, nq + 2 * nkv, d)

    def norm_rot(h, gain, pos):
        if gain is not None:
            h = h * torch.rsqrt((h * h).mean(-1, keepdim=True) + eps) * gain.double()
        if not rope:
            return h
        c, s = torch.cos(ang[pos])[:, None, :], torch.sin(ang[pos])[:, None, :]
        a, b = h[..., :d // 2], h[..., d // 2:]
        return torch.cat([a * c - b * s, a * s + b * c], dim=-1)

    pos_t = torch.tensor(positions)
    ref_q = norm_rot(y[:, :nq], qg, pos_t)
    ref_k = norm_rot(y[:, nq:nq + nkv], kg, pos_t)
    ref_v = y[:, nq + nkv:]
    tol = 2e-2    # bfloat16 output of values up to about 4
    assert float((q_out.double().cpu().reshape(M, nq, d) - ref_q).abs().max()) < tol
    if not write:
        assert float(kp.abs().sum()) == 0 and float(vp.abs().sum()) == 0
        return
    pages = table[torch.tensor(token_req), pos_t // ps].long()
    rows = pos_t % ps
    assert float((kp.cpu()[pages, :, rows].double() - ref_k).abs().max()) < tol
    assert float((vp.cpu()[pages, :, rows].double() - ref_v).abs().max()) < tol
    assert int((kp.abs().sum(dim=(1, 3)) > 0).sum()) == M            # nothing else was touched


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq, nkv, d, rot, ps", [(4, 2, 16, 16, 4), (6, 3, 48, 48, 32), (8, 1, 128, 128, 64),
                                                (3, 3, 34, 34, 5), (4, 2, 32, 16, 8)])
def test_qk_norm_rope_kv(dtype, nq, nkv, d, rot, ps):
    torch.manual_seed(6)
    n, theta, eps = 9, 5e4, 1e-5
    positions = [3, 4, 5, 0, 17, 18, 19, 20, 63]
    token_req = [0, 0, 0, 1, 2, 2, 2, 2, 2]
    qkv = torch.randn(n, (nq + 2 * nkv) * d).to(dtype)
    qg, kg = 1 + 0.1 * torch.randn(d), 1 + 0.1 * torch.randn(d)
    inv_freq = torch.pow(torch.tensor(theta), -(2.0 * torch.arange(rot // 2)) / rot)
    cos, sin = _k().rope_table(inv_freq.to(DEV), 64)
    ang = torch.arange(64, dtype=torch.float32)[:, None] * inv_freq[None, :]
    assert float((cos.cpu() - torch.cos(ang)).abs().max()) < 2e-6 and float((sin.cpu() - torch.sin(ang)).abs().max()) < 2e-6
    max_blocks = -(-64 // ps)
    num_pages = 3 * max_blocks + 2
    table = torch.full((3, max_blocks), -1, dtype=torch.int32)
    perm = torch.randperm(num_pages).tolist()
    for r in range(3):
        for b in range(max_blocks):
            table[r, b] = perm.pop()
    kp = torch.zeros(num_pages, nkv, ps, d, dtype=dtype, device=DEV)
    vp = torch.zeros_like(kp)
    q_out = torch.empty(n, nq * d, dtype=dtype, device=DEV)
    st = _status()
    _k().qk_norm_rope_kv(qkv.to(DEV), q_out, qg.to(DEV), kg.to(DEV), eps, cos, sin, rot, I(positions), I(token_req),
                         table.to(DEV), ps, kp, vp, nq, nkv, d, st)
    assert st.item() == 0

    def norm_rot(x, gain, pos):
        x = x.double()
        x = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * gain.double()
        half = rot // 2
        c, s = torch.cos(ang[pos].double()), torch.sin(ang[pos].double())
        a, b = x[..., :half], x[..., half:rot]
        return torch.cat([a * c - b * s, a * s + b * c, x[..., rot:]], dim=-1)

    tol = 1e-5 if dtype == torch.float32 else 3e-2
    x = qkv.reshape(n, nq + 2 * nkv, d)
    for t in range(n):
        ref_q = norm_rot(x[t, :nq], qg, positions[t])
        assert float((q_out[t].double().cpu().reshape(nq, d) - ref_q).abs().max()) < tol
        page, row = int(table[token_req[t], positions[t] // ps]), positions[t] % ps
        ref_k = norm_rot(x[t, nq:nq + nkv], kg, positions[t])
        assert float((kp[page, :, row].double().cpu() - ref_k).abs().max()) < tol
        assert torch.equal(vp[page, :, row].cpu(), x[t, nq + nkv:])          # values are stored as they are
    written = {(int(table[token_req[t], positions[t] // ps]), positions[t] % ps) for t in range(n)}
    assert int((kp.abs().sum(dim=(1, 3)) > 0).sum()) == len(written)          # nothing else was touched


# ------------------------------------------------------------------ attention

def _attention_case(nq, nkv, d, ctx, new, ps, window, dtype, mode, decode_chunk=0, key_ranges=None, in_ulps=False):
    """ctx[r] cached positions and new[r] query tokens per request. One query per request
    has a far key that dominates its softmax, so a missed or misplaced key changes the result.
    Returns the largest absolute error, or with `in_ulps` the largest error in units of
    (6e-3 + half a bfloat16 step of the value), which does not grow with the value."""
    torch.manual_seed(7)
    k = _k()
    R = len(ctx)
    tot = [c + n for c, n in zip(ctx, new)]
    k_seq = [torch.randn(t, nkv, d).to(dtype).float() for t in tot]
    v_seq = [torch.randn(t, nkv, d).to(dtype).float() for t in tot]
    n = sum(new)
    q = (torch.randn(n, nq * d) * 1.5).to(dtype).float()
    positions, token_req, q_start = [], [], [0]
    for r in range(R):
        positions += list(range(ctx[r], tot[r]))
        token_req += [r] * new[r]
        q_start.append(q_start[-1] + new[r])
    for r in range(R):
        t = q_start[r + 1] - 1
        far = max(0, tot[r] - window) if window else min(1, tot[r] - 1)   # the window's far edge, or nearly the first key
        q[t, :d] = 0
        q[t, 0] = 8.0
        k_seq[r][far, 0, :] = 0
        k_seq[r][far, 0, 0] = 8.0
    num_pages = sum(-(-t // ps) for t in tot) + 3
    kp, vp, table = build_pages(k_seq, v_seq, ps, num_pages, nkv, d, dtype, DEV)
    scale = d ** -0.5
    ref = ref_paged_attention(q, k_seq, v_seq, positions, token_req, nq, nkv, d, scale, window)
    qd = q.to(dtype).to(DEV)
    out = torch.zeros_like(qd)
    st = _status()
    if mode == "generic":
        k.attention_generic(qd, out, kp, vp, table, I(positions), I(token_req), nq, nkv, d, scale, window, st)
    elif mode.startswith("decode"):
        chunk, splits = k.attention_decode_plan(R, nkv, max(tot) + 70)
        if decode_chunk:
            chunk, splits = decode_chunk, -(-(max(tot) + 70) // decode_chunk)
        k.attention_decode(qd, out, kp, vp, table, I(tot), I(q_start), nq, nkv, d, scale, window, chunk, splits, st,
                           use_tma=mode.endswith("tma"))
    else:
        tiles = [(r, q_start[r] + t0) for r in range(R) for t0 in range(0, new[r], k.QUERY_TILE)]
        impl = {"prefill": "cpasync", "prefill_tma": "tma", "prefill_tcgen05": "tcgen05"}[mode]
        k.attention_prefill(qd, out, kp, vp, table, I(q_start), I(ctx), I([t[0] for t in tiles]),
                            I([t[1] for t in tiles]), nq, nkv, d, scale, window, st, impl=impl, key_ranges=key_ranges)
    assert st.item() == 0
    err = (out.double().cpu() - ref).abs()
    if in_ulps:
        return float((err / (6e-3 + ref.abs() * 2.0 ** -8)).max())
    return float(err.max())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq, nkv, d, ctx, new, ps, window", [
    (4, 2, 16, [0, 5], [33, 1], 4, 0), (6, 3, 48, [40, 0], [7, 100], 32, 0), (8, 1, 32, [300], [3], 8, 0),
    (4, 4, 80, [0], [70], 16, 0), (8, 2, 128, [200, 0], [2, 130], 64, 0), (2, 1, 256, [30], [10], 16, 0),
    (6, 3, 64, [40, 0], [90, 150], 32, 50), (4, 2, 16, [100], [1], 7, 9),
])
def test_attention_generic(dtype, nq, nkv, d, ctx, new, ps, window):
    err = _attention_case(nq, nkv, d, ctx, new, ps, window, dtype, "generic")
    assert err < (2e-5 if dtype == torch.float32 else 1.2e-2)


@pytest.mark.parametrize("mode", ["prefill", "prefill_tma"])
@pytest.mark.parametrize("nq, nkv, d, ctx, new, ps, window", [
    (4, 2, 64, [0], [64], 16, 0), (4, 2, 64, [0, 0], [100, 3], 16, 0), (8, 2, 128, [0, 37, 200], [130, 64, 1], 64, 0),
    (8, 1, 128, [5, 300], [70, 2], 8, 0), (6, 3, 64, [40, 0], [90, 150], 32, 50), (8, 2, 128, [100, 0], [300, 257], 128, 0),
    (16, 1, 64, [129], [127], 32, 0),
])
def test_attention_prefill_kernels(mode, nq, nkv, d, ctx, new, ps, window):
    assert _attention_case(nq, nkv, d, ctx, new, ps, window, torch.bfloat16, mode) < 1.2e-2


@pytest.mark.parametrize("nq, nkv, ctx, new, ps, window", [
    (8, 2, [0], [128], 64, 0), (8, 2, [0], [17], 64, 0), (8, 2, [0, 37, 200], [130, 64, 1], 64, 0), (8, 1, [5, 300], [70, 2], 8, 0),
    (8, 2, [100, 0], [300, 257], 128, 0), (4, 4, [40, 0], [90, 150], 32, 50), (32, 8, [0], [1024], 64, 0), (2, 1, [700], [129], 16, 100),
])
def test_attention_prefill_tcgen05(nq, nkv, ctx, new, ps, window):
    """The tensor-memory kernel (head size 128): spans that end inside a tile, several requests, page
    pieces smaller and larger than a tile, a window, an odd number of key tiles (the two softmax groups
    then hold different numbers of tiles)."""
    assert _attention_case(nq, nkv, 128, ctx, new, ps, window, torch.bfloat16, "prefill_tcgen05") < 1.2e-2


@pytest.mark.parametrize("ranges, ctx, new, ps, window", [
    (2, [0], [300], 64, 0), (3, [1000, 0], [130, 257], 64, 0), (4, [40], [64], 16, 0),   # the last: more ranges than key tiles
    (8, [2100], [200], 128, 0), (3, [700], [129], 32, 500), (2, [0, 37, 200], [130, 64, 1], 8, 0),
])
def test_attention_prefill_tcgen05_key_ranges(ranges, ctx, new, ps, window):
    """The keys of every query tile cut into ranges over separate CTAs and merged by a second kernel:
    ranges that are empty for short rows, a window that leaves the first ranges without keys."""
    assert _attention_case(8, 2, 128, ctx, new, ps, window, torch.bfloat16, "prefill_tcgen05", key_ranges=ranges) < 1.2e-2
    k = _k()
    # a launch that fills its rounds stays whole; one of few CTAs and many keys is cut
    assert k.attention_prefill_ranges(512, 2048) == 1 and k.attention_prefill_ranges(512, 8192) == 1 and k.attention_prefill_ranges(512, 32768) == 1
    assert k.attention_prefill_ranges(296, 30000) == 1
    assert k.attention_prefill_ranges(128, 2560) == 1 and k.attention_prefill_ranges(128, 6656) == 2 and k.attention_prefill_ranges(128, 31232) == 2
    assert k.attention_prefill_ranges(32, 32768) == 8


@pytest.mark.parametrize("seed", [11, 12])
def test_attention_prefill_tcgen05_random_cases(seed):
    """Twenty drawn cases a seed: heads and groups, several requests with and without earlier
    context, spans of one token to several query tiles, every page size, windows, key ranges."""
    import random

    rng = random.Random(seed)
    for case in range(20):
        nkv = rng.choice([1, 2, 4, 8])
        nq = nkv * rng.choice([1, 2, 4, 5, 8])
        n_req = rng.choice([1, 1, 2, 3, 4])
        ps = rng.choice([8, 16, 32, 64, 128, 256])
        ctx = [rng.choice([0, 0, rng.randint(1, 200), rng.randint(200, 3000)]) for _ in range(n_req)]
        new = [rng.choice([1, 2, rng.randint(3, 130), rng.randint(130, 700)]) for _ in range(n_req)]
        window = rng.choice([0, 0, 0, rng.randint(1, 600)])
        ranges = rng.choice([None, None, 1, 2, 3, 4, 8])
        err = _attention_case(nq, nkv, 128, ctx, new, ps, window, torch.bfloat16, "prefill_tcgen05", key_ranges=ranges, in_ulps=True)
        assert err < 1.0, (case, nq, nkv, ctx, new, ps, window, ranges, err)      # measured: 0.73 at most


def test_attention_prefill_without_tma_takes_any_page_size():
    assert _attention_case(4, 2, 64, [10, 0], [90, 31], 24, 0, torch.bfloat16, "prefill") < 1.2e-2
    assert _attention_case(4, 2, 64, [10, 77], [1, 1], 24, 0, torch.bfloat16, "decode") < 1.2e-2


@pytest.mark.parametrize("mode", ["decode", "decode_tma"])
@pytest.mark.parametrize("nq, nkv, d, ctx, ps, window", [
    (4, 2, 64, [63], 16, 0), (4, 2, 64, [10, 200, 64], 16, 0), (32, 8, 128, [2047, 100, 513, 0], 64, 0),
    (8, 1, 128, [700, 3], 8, 0), (8, 2, 128, [300, 90], 32, 64), (8, 2, 128, [1000, 90], 256, 0),
])
def test_attention_decode_kernels(mode, nq, nkv, d, ctx, ps, window):
    assert _attention_case(nq, nkv, d, ctx, [1] * len(ctx), ps, window, torch.bfloat16, mode) < 1.2e-2


@pytest.mark.parametrize("chunk, ctx, window", [
    (2048, [2047, 100, 513, 0], 0),     # one range: the CTA writes the result itself
    (2048, [2047, 100, 513, 0], 300),   # the same with a window
    (1024, [1500, 100, 1023, 1024], 0), # two ranges; a request of two key tiles has one in each
    (512, [1999, 64, 700, 0], 0),       # five ranges
    (256, [1700, 300, 255, 256], 200),  # a window: its tiles are dealt out over the ranges, the rest are empty
    (192, [1700, 300, 255, 256], 0),    # ten ranges
])
def test_attention_decode_key_ranges(chunk, ctx, window):
    """One key range per request (the kernel writes the output itself) and several (partial results,
    merged by a second kernel). A request's key tiles are dealt out evenly over the ranges, so a request
    with fewer tiles than ranges leaves the last ranges empty."""
    assert _attention_case(8, 2, 128, ctx, [1] * len(ctx), 64, window, torch.bfloat16, "decode_tma", decode_chunk=chunk) < 1.2e-2
    assert _attention_case(4, 1, 64, ctx[:2], [1, 1], 16, window, torch.bfloat16, "decode_tma", decode_chunk=chunk) < 1.2e-2


@pytest.mark.parametrize("nq, nkv, d, lens, ps, window, chunk, partial, writes", [
    (8, 2, 128, [1, 64, 65, 300, 513], 64, 0, 0, True, True),      # the new key opens a page, ends one, lies inside
    (8, 2, 128, [1, 64, 65, 300, 513], 16, 0, 128, False, True),   # several ranges: only the last one holds the new key
    (4, 4, 64, [33, 200], 8, 0, 64, True, True),
    (6, 1, 64, [90, 7, 129], 32, 50, 0, False, True),              # a window
    (8, 2, 128, [10, 140], 64, 0, 0, True, False),                 # the cache is another layer's: nothing is written
    (32, 8, 128, [2049] * 3, 64, 0, 0, True, True),
])
def test_attention_decode_with_rope_equals_the_two_kernels(nq, nkv, d, lens, ps, window, chunk, partial, writes):
    """One launch that makes the queries and the new key and value from the q/k/v projection against
    qk_norm_rope_kv followed by attention_decode (each checked against its formulas above): the same
    output, the same cache rows, nothing else touched."""
    torch.manual_seed(len(lens) * 7 + d)
    k = _k()
    B, eps = len(lens), 1e-6
    width = (nq + 2 * nkv) * d
    y = torch.randn(B, width, device=DEV)
    if partial:
        parts = torch.randn(3, B, width, device=DEV)
        parts[2] = y - parts[0] - parts[1]
        qkv = parts.contiguous()
    else:
        qkv = y.bfloat16()
    qg, kg = (1 + 0.1 * torch.randn(d)).to(DEV), (1 + 0.1 * torch.randn(d)).to(DEV)
    inv_freq = torch.pow(torch.tensor(1e4), -(2.0 * torch.arange(d // 2)) / d)
    cos, sin = k.rope_table(inv_freq.to(DEV), max(lens) + 1)
    max_blocks = -(-max(lens) // ps) + 1
    num_pages = B * max_blocks + 2
    perm = torch.randperm(num_pages).tolist()
    table = torch.tensor([[perm.pop() for _ in range(max_blocks)] for _ in range(B)], dtype=torch.int32, device=DEV)
    pages = [(torch.randn(num_pages, nkv, ps, d, device=DEV) * 0.7).bfloat16() for _ in range(2)]
    kv_len, q_start = I(lens), I(list(range(B + 1)))
    positions, token_req = I([n - 1 for n in lens]), I(list(range(B)))
    plan = k.attention_decode_plan(B, nkv, max(lens) + 40)
    if chunk:
        plan = (chunk, -(-(max(lens) + 40) // chunk))
    # the two kernels
    kp1, vp1 = pages[0].clone(), pages[1].clone()
    q = torch.empty(B, nq * d, dtype=torch.bfloat16, device=DEV)
    st = _status()
    if writes:
        k.qk_norm_rope_kv(qkv, q, qg, kg, eps, cos, sin, d, positions, token_req, table, ps, kp1, vp1, nq, nkv, d, st)
    else:
        k.qk_norm_rope_kv(qkv, q, qg, kg, eps, cos, sin, d, positions, token_req, table, ps, None, None, nq, nkv, d, st)
    out1 = torch.empty_like(q)
    k.attention_decode(q, out1, kp1, vp1, table, kv_len, q_start, nq, nkv, d, d ** -0.5, window, plan[0], plan[1], st, use_tma=True)
    # the one kernel
    kp2, vp2 = pages[0].clone(), pages[1].clone()
    out2 = torch.empty_like(q)
    k.attention_decode_rope(qkv, out2, qg, kg, eps, cos, sin, kp2, vp2, writes, table, kv_len, q_start, nq, nkv, d, d ** -0.5,
                            window, plan[0], plan[1], st)
    assert st.item() == 0
    assert float((out1.float() - out2.float()).abs().max()) < 4e-3
    assert float((kp1.float() - kp2.float()).abs().max()) < 2e-2 and float((vp1.float() - vp2.float()).abs().max()) < 2e-2
    changed = int(((kp2 != pages[0]).sum(dim=3) > 0).sum())
    assert changed == (B * nkv if writes else 0)


def test_attention_kernels_refuse_what_they_do_not_cover():
    from quantinfer_b200.errors import KernelError

    k = _k()
    assert not k.attention_mma_supported(4, 2, 48) and not k.attention_tma_supported(4, 2, 64, 24)
    q = torch.zeros(1, 4 * 48, dtype=torch.bfloat16, device=DEV)
    pages = torch.zeros(2, 2, 16, 48, dtype=torch.bfloat16, device=DEV)
    with pytest.raises(KernelError, match="not covered"):
        k.attention_prefill(q, torch.empty_like(q), pages, pages, I([[0]]), I([0, 1]), I([0]), I([0]), I([0]), 4, 2, 48,
                            1.0, 0, _status(), use_tma=False)
    with pytest.raises(KernelError, match="limit"):
        big = torch.zeros(1, 2 * 272, dtype=torch.float32, device=DEV)
        k.attention_generic(big, torch.empty_like(big), torch.zeros(1, 2, 4, 272, device=DEV),
                            torch.zeros(1, 2, 4, 272, device=DEV), I([[0]]), I([0]), I([0]), 2, 2, 272, 1.0, 0, _status())


# ------------------------------------------------------------------ activation, sampling

@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("interleaved", [False, True])
def test_silu_mul(dtype, interleaved):
    torch.manual_seed(8)
    g, u = torch.randn(5, 57).to(dtype) * 3, torch.randn(5, 57).to(dtype)
    gu = torch.stack([g, u], dim=2).reshape(5, 114) if interleaved else torch.cat([g, u], dim=1)
    out = torch.empty(5, 57, dtype=dtype, device=DEV)
    _k().silu_mul(gu.contiguous().to(DEV), out, interleaved=interleaved)
    ref = g.double() / (1 + torch.exp(-g.double())) * u.double()
    assert float((out.double().cpu() - ref).abs().max()) < (1e-6 if dtype == torch.float32 else 3e-2)


def _sample(logits, temperature=None, top_k=None, top_p=None, seed=None, counter=None):
    rows = logits.shape[0]
    st = _status()
    out = torch.empty(rows, dtype=torch.int32, device=DEV)
    f = lambda v, dt: None if v is None else torch.tensor(v, dtype=dt, device=DEV)
    _k().sample(logits.to(DEV), f(temperature, torch.float32), f(top_k, torch.int32), f(top_p, torch.float32),
                f(seed, torch.int64), f(counter, torch.int32), out, st)
    return out.cpu().tolist(), st.item()


def test_sample_greedy_first_maximum():
    x = torch.randn(4, 1000)
    x[1, 17] = x[1, 900] = 50.0          # a tie: the lowest index wins
    x[2, 999] = 60.0
    toks, st = _sample(x)
    assert st == 0 and toks == [int(x[0].argmax()), 17, 999, int(x[3].argmax())]
    x[3, 5] = float("nan")
    assert _sample(x)[1] == _k().STATUS_NON_FINITE


@pytest.mark.parametrize("vocab", [50, 517, 4099])
def test_sample_matches_the_plain_sampler(vocab):
    torch.manual_seed(9)
    rows = 24
    x = torch.randn(rows, vocab) * 2
    x[:, 3] = x[:, 11]                    # ties inside the candidate set
    temps = [0.0, 0.8, 1.3, 0.5] * 6
    ks = [0, 0, 5, 20, 0, 1] * 4
    ps = [0.0, 0.0, 0.0, 0.0, 0.9, 0.5, 0.3, 1.0] * 3
    seeds = [7 + (r << 33) for r in range(rows)]
    counters = list(range(rows))
    toks, st = _sample(x, temps, ks, ps, seeds, counters)
    assert st == 0
    for r in range(rows):
        expect = plain_sample(x[r], temps[r], ks[r] or None, ps[r] or None, seeds[r], counters[r])
        assert toks[r] == expect, (r, temps[r], ks[r], ps[r])


def test_sample_follows_the_distribution_and_the_counter():
    x = torch.tensor([[0.0, 2.0, 1.0, -1.0, 2.0]]).repeat(4000, 1)
    toks, _ = _sample(x, [1.0] * 4000, None, None, [12345] * 4000, list(range(4000)))
    p = torch.softmax(x[0], 0)
    freq = torch.bincount(torch.tensor(toks), minlength=5).double() / 4000
    assert float((freq - p.double()).abs().max()) < 0.03
    again, _ = _sample(x[:50], [1.0] * 50, None, None, [12345] * 50, list(range(50)))
    assert again == toks[:50]            # same seed and counter, same token
    other, _ = _sample(x[:50], [1.0] * 50, None, None, [12346] * 50, list(range(50)))
    assert other != toks[:50]


@pytest.mark.parametrize("vocab", [517, 4099])
def test_sample_from_slot_records(vocab):
    """The options of a row come from its request's slot record, found through the step's arrays
    (row -> flat token -> entry -> slot), and the kernel advances the record's counter: three draws in a
    row equal the plain sampler's with counters c, c + 1, c + 2, for requests that sit in other slots
    than their place in the batch, greedy rows among them."""
    from quantinfer_b200.sampling import GenerationConfig, RequestSlots

    torch.manual_seed(3)
    slots = RequestSlots(8, DEV)
    cfgs = {5: GenerationConfig(temperature=0.8, seed=11), 2: GenerationConfig(temperature=1.2, top_k=20, seed=(1 << 40) + 5),
            7: GenerationConfig(), 0: GenerationConfig(temperature=0.6, top_p=0.7, seed=3)}
    start = {5: 0, 2: 9, 7: 4, 0: 100}
    for slot, cfg in cfgs.items():
        slots.assign(slot, cfg, start[slot])
    # a step of four entries with 3, 1, 2 and 1 tokens; the rows wanted are the last token of each
    slot_ids, token_req, logit_rows = I([5, 2, 7, 0]), I([0, 0, 0, 1, 2, 2, 3]), I([2, 3, 5, 6])
    order = [5, 2, 7, 0]
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    for draw in range(3):
        x = torch.randn(4, vocab) * 2
        out = torch.empty(4, dtype=torch.int32, device=DEV)
        _k().sample_slots(x.to(DEV), logit_rows, token_req, slot_ids, slots.table, False, out, st)
        for r, slot in enumerate(order):
            c = cfgs[slot]
            assert int(out[r]) == plain_sample(x[r], c.temperature, c.top_k, c.top_p, c.seed, start[slot] + draw), (draw, slot)
    assert int(st) == 0
    assert slots.table[:, 3].tolist() == [103, 0, 12, 0, 0, 3, 0, 7]        # every record's counter moved by three
    # a step that the host knows to be all greedy takes the other kernel; the counter still moves
    slots.assign(1, GenerationConfig(), 0)
    x = torch.randn(1, vocab)
    out = torch.empty(1, dtype=torch.int32, device=DEV)
    _k().sample_slots(x.to(DEV), I([0]), I([0]), I([1]), slots.table, True, out, st)
    assert int(out[0]) == int(x[0].argmax()) and int(slots.table[1, 3]) == 1
    assert slots.table[1].tolist()[6:] == [128, -1]                          # max_new_tokens, no eos


def test_advance_decode():
    tok, pos, sp, kv, ctr = I([5, 6]), I([10, 20]), I([10, 20]), I([11, 21]), I([0, 3])
    hist = torch.zeros(2, dtype=torch.int32, device=DEV)
    _k().advance_decode(tok, pos, sp, kv, ctr, I([77, 88]), hist)
    assert tok.tolist() == [77, 88] and pos.tolist() == [11, 21] and sp.tolist() == [11, 21]
    assert kv.tolist() == [12, 22] and ctr.tolist() == [1, 4] and hist.tolist() == [77, 88]


# ------------------------------------------------------------------ lengths that a launch does not cover are flagged


def test_lengths_beyond_what_a_launch_covers_set_a_status_bit():
    """A position beyond the rotation table, and keys beyond the key ranges of a decode launch: the
    kernels read nothing out of range and drop nothing silently, they set STATUS_BAD_RANGE (the engine
    never passes such lengths; an embedder of the C symbols might)."""
    k = _k()
    torch.manual_seed(1)
    nq, nkv, d, ps = 4, 2, 64, 16
    # (1) the rotation table has 32 rows, one token stands at position 40
    inv_freq = torch.pow(torch.tensor(1e4), -(2.0 * torch.arange(d // 2)) / d)
    cos, sin = k.rope_table(inv_freq.to(DEV), 32)
    qkv = torch.randn(2, (nq + 2 * nkv) * d, device=DEV)
    q_out = torch.empty(2, nq * d, device=DEV)
    table = I([[0, 1, 2, 3]])
    kp = torch.zeros(4, nkv, ps, d, device=DEV)
    vp = torch.zeros_like(kp)
    for positions, want in (([3, 31], 0), ([3, 40], k.STATUS_BAD_RANGE)):
        st = _status()
        k.qk_norm_rope_kv(qkv, q_out, None, None, 1e-6, cos, sin, d, I(positions), I([0, 0]), table, ps, kp, vp, nq, nkv, d, st)
        assert st.item() == want, positions
    assert torch.isfinite(q_out).all()
    # (2) two key ranges of 64 keys cover 128 positions; one request holds 200
    ctx = [100, 200]
    max_blocks = -(-max(ctx) // ps)
    pages = torch.randn(2 * max_blocks, nkv, ps, d, device=DEV).bfloat16()
    tbl = torch.arange(2 * max_blocks, dtype=torch.int32, device=DEV).view(2, max_blocks)
    q = torch.randn(2, nq * d, device=DEV).bfloat16()
    out = torch.empty_like(q)
    for use_tma in (True, False):
        for n_splits, want in ((4, 0), (2, k.STATUS_BAD_RANGE)):
            st = _status()
            k.attention_decode(q, out, pages, pages, tbl, I(ctx), I([0, 1, 2]), nq, nkv, d, d ** -0.5, 0, 64, n_splits, st,
                               use_tma=use_tma)
            assert st.item() == want, (use_tma, n_splits)
    assert k.status_names(k.STATUS_BAD_RANGE) and "rotation table" in k.status_names(k.STATUS_BAD_RANGE)[0]


# ------------------------------------------------------------------ kernels in 16-byte pieces beside their element-wise forms

def _off(t):
    """The same numbers in a buffer that starts off every 16-byte boundary: the kernels fall back to one element at a time."""
    return torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape).copy_(t)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n, h", [(1, 8), (3, 136), (700, 2048)])
def test_pieces_dyt_and_act_mul(dtype, n, h):
    torch.manual_seed(h)
    r, y, f = torch.randn(n, h, device=DEV), torch.randn(3, n, h, device=DEV), [torch.randn(h, device=DEV) for _ in range(5)]
    a = [torch.full((1,), v, device=DEV) for v in (0.7, 1.3)]
    got = []
    for c in (lambda t: t, _off):
        for parts in (y, y[0].to(dtype)):
            resid, out = c(r.clone()), c(torch.empty(n, h, device=DEV, dtype=dtype))
            _k().dyt(resid, c(parts), f[0], (c(f[1]), f[2], a[0]), 0.6, (f[3], f[4], a[1]), out)
            got += [resid, out]
        for name in ("silu", "gelu", "gelu_tanh", "relu", "relu2", "tanh"):
            for inter in (False, True):
                act = c(torch.empty(n, h, device=DEV, dtype=dtype))
                _k().act_mul(c(y[:2].reshape(n, 2 * h).to(dtype)), act, name, interleaved=inter)
                got.append(act)
    for fast, slow in zip(got[:len(got) // 2], got[len(got) // 2:]):      # a product and a sum may be one rounding in one form and two in the other
        tol = 2e-6 if fast.dtype == torch.float32 else 2.0 ** -7
        assert bool(((fast.float() - slow.float()).abs() <= tol * (1 + slow.float().abs())).all())


@pytest.mark.parametrize("gate", ["silu_before", "silu", "sigmoid", "plain"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n, groups, gw", [(2, 1, 8), (5, 3, 264), (3, 1, 8192), (2, 2, 8200), (1, 1, 16392), (1, 1, 32768)])
def test_pieces_gated_group_rmsnorm(n, groups, gw, dtype, gate):
    torch.manual_seed(gw)
    y, z, gain = torch.randn(n, groups * gw, device=DEV), torch.randn(n, groups * gw, device=DEV).to(dtype), torch.randn(groups * gw, device=DEV)
    fast, slow = torch.empty(n, groups * gw, device=DEV), _off(torch.empty(n, groups * gw, device=DEV))
    _k().gated_group_rmsnorm(y, z, gain, 1e-5, fast, groups, gate, 0.5)
    _k().gated_group_rmsnorm(y, z, gain, 1e-5, slow, groups, gate, 0.5)
    # another order of a sum of squares of up to 32,768 numbers, and a gate that is rounded in another place: a few roundings
    assert bool(((fast - slow).abs() <= 1e-5 * slow.abs() + 1e-7).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq, nkv, d, dv, rot, inter, norm", [
    (4, 2, 16, 16, 16, False, False), (4, 1, 64, 40, 32, False, True), (8, 2, 128, 128, 64, False, False), (3, 3, 128, 128, 128, False, True),
    (2, 1, 256, 256, 256, False, False), (4, 2, 64, 64, 0, False, False), (4, 2, 128, 64, 64, True, True), (2, 1, 200, 8, 48, False, True),
])
@pytest.mark.parametrize("biased", [False, True])
def test_pieces_bias_rope_kv(dtype, nq, nkv, d, dv, rot, inter, norm, biased):
    torch.manual_seed(d + rot)
    n, page = 37, 16
    total = (nq + nkv) * d + nkv * dv
    proj, bias = torch.randn(n, total, device=DEV).to(dtype), torch.randn(total, device=DEV) if biased else None
    freq = torch.rand(rot // 2, device=DEV) if rot else None
    gains = (torch.randn(d, device=DEV), torch.randn(d, device=DEV)) if norm else (None, None)
    pos, req, table = I([3 * i for i in range(n)]), I([0] * n), I([list(range(8))])
    got = []
    for c in (lambda t: t, _off):
        q, st = torch.zeros(n, nq * d, device=DEV, dtype=dtype), _status()
        k, v = torch.zeros(8, nkv, page, d, device=DEV, dtype=dtype), torch.zeros(8, nkv, page, dv, device=DEV, dtype=dtype)
        _k().bias_rope_kv(c(proj), bias, q, freq, rot, inter, pos, req, table, page, k, v, nq, nkv, d, dv, st, q_gain=gains[0], k_gain=gains[1],
                          norm_eps=1e-6 if norm else 0.0, head_norm=norm)
        got.append((q, k, v))
        assert int(st) == 0
    for fast, slow in zip(*got):      # the head's sum of squares in another order; a result in bfloat16 may round to the other side
        assert bool(((fast.float() - slow.float()).abs() <= (2e-6 if dtype == torch.float32 else 2.0 ** -7) * (1 + slow.float().abs())).all())


@pytest.mark.parametrize("E", [4, 32, 33, 64, 65, 128, 129, 256, 257, 1000])
def test_moe_route_and_group_over_the_numbers_of_experts(E):
    torch.manual_seed(E)
    k, n, top = _k(), 301, 4
    z, corr = torch.randn(n, E, device=DEV), torch.randn(E, device=DEV) * 0.01
    ids, w = torch.empty(n, top, dtype=torch.int32, device=DEV), torch.empty(n, top, device=DEV)
    k.moe_route(z, corr, ids, w, 1.5)
    s = torch.softmax(z.double(), 1)
    chosen = (s + corr.double()).topk(top, 1).indices
    assert torch.equal(ids.long().sort(1).values, chosen.sort(1).values)
    ref = s.gather(1, ids.long())
    assert torch.allclose(w.double(), 1.5 * ref / ref.sum(1, keepdim=True), rtol=1e-5)
    off, order, place = I([0] * (E + 1)), I([0] * (n * top)), I([0] * (n * top))
    rows = k.moe_tile_rows()
    tiles = torch.empty((min(n * top, n * top // rows + E), 3), dtype=torch.int32, device=DEV)
    k.moe_group(ids, E, off, order, place, tiles)
    count = torch.bincount(ids.flatten().long(), minlength=E)
    assert torch.equal(off[1:].long(), count.cumsum(0)) and int(off[0]) == 0
    assert torch.equal(place[order.long()].long(), torch.arange(n * top, device=DEV))
    assert torch.equal(ids.flatten()[order.long()].long(), torch.repeat_interleave(torch.arange(E, device=DEV), count))
    want = [(e, int(off[e]) + r, min(rows, int(count[e]) - r)) for e in range(E) for r in range(0, int(count[e]), rows)]
    assert [tuple(t) for t in tiles.tolist() if t[0] >= 0] == want
