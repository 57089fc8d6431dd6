"""Each CUDA kernel alone against a plain float64 reference, at sizes other than the engine's."""
import math

import pytest
import torch

import qwen3_plain as P

pytestmark = pytest.mark.gpu

BF16, F32 = torch.bfloat16, torch.float32
TOL = {F32: 2e-6, BF16: 1.2e-2}     # relative to the largest reference magnitude


def _close(got, ref, dtype, scale=1.0):
    err = float((got.double().cpu() - ref.double().cpu()).abs().max())
    mag = float(ref.double().abs().max()) or 1.0
    assert err <= TOL[dtype] * scale * mag, f"error {err:.3g} vs magnitude {mag:.3g}"


def _err(dev):
    return torch.zeros(1, dtype=torch.int32, device=dev)


def test_launches_go_to_the_current_stream(cuda_device, monkeypatch):
    from binfer_b200.csrc import ops
    for _ in range(2):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            assert ops._stream().value == s.cuda_stream
        assert (ops._stream().value or 0) == torch.cuda.current_stream().cuda_stream
        monkeypatch.setattr(ops, "_raw_stream", None)      # a torch without the private name


# ------------------------------------------------------------------ elementwise
@pytest.mark.parametrize("dtype", [F32, BF16])
def test_embed_gather(cuda_device, dtype):
    from binfer_b200.csrc import ops
    table = torch.randn(301, 100, device=cuda_device).to(dtype)
    ids = torch.tensor([0, 300, 17, 17, 5], dtype=torch.int32, device=cuda_device)
    out = torch.empty(5, 100, device=cuda_device)
    err = _err(cuda_device)
    ops.embed_gather(table, ids, out, 1.0, err)
    assert torch.equal(out, table.float()[ids.long()])
    assert int(err.item()) == 0
    bad = torch.tensor([3, 301], dtype=torch.int32, device=cuda_device)
    out2 = torch.ones(2, 100, device=cuda_device)
    ops.embed_gather(table, bad, out2, 1.0, err)
    assert int(err.item()) == 1 and float(out2[1].abs().max()) == 0.0


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("H", [100, 1536, 5000])
def test_add_rmsnorm(cuda_device, dtype, H):
    from binfer_b200.csrc import ops
    resid = torch.randn(9, H, device=cuda_device)
    delta = torch.randn(9, H, device=cuda_device).to(dtype)
    w = 1 + 0.1 * torch.randn(H, device=cuda_device)
    r0 = resid.clone()
    out = torch.empty(9, H, device=cuda_device, dtype=dtype)
    ops.add_rmsnorm(resid, delta, w, out, 1e-5)
    x = r0.double() + delta.double()
    _close(resid, x, F32)
    _close(out, P.rms_norm(x, w.double(), 1e-5), dtype)
    # selected rows, no pending add, stream untouched
    rows = torch.tensor([8, 2], dtype=torch.int32, device=cuda_device)
    keep = resid.clone()
    out2 = torch.empty(2, H, device=cuda_device, dtype=dtype)
    ops.add_rmsnorm(resid, None, w, out2, 1e-6, rows=rows, write_back=False)
    assert torch.equal(resid, keep)
    _close(out2, P.rms_norm(keep.double()[[8, 2]], w.double(), 1e-6), dtype)


@pytest.mark.parametrize("dtype", [F32, BF16])
def test_silu_mul_and_residual_add(cuda_device, dtype):
    from binfer_b200.csrc import ops
    gu = (3 * torch.randn(7, 2 * 150, device=cuda_device)).to(dtype)
    out = torch.empty(7, 150, device=cuda_device, dtype=dtype)
    ops.silu_mul(gu, out)
    g, u = gu.double()[:, :150], gu.double()[:, 150:]
    _close(out, g / (1 + torch.exp(-g)) * u, dtype)
    resid = torch.randn(7, 150, device=cuda_device)
    want = resid.double() + out.double()
    ops.residual_add(resid, out)
    _close(resid, want, F32)


@pytest.mark.parametrize("M", [1, 7, 16, 63, 65, 130])
def test_sgemm_true_float32(cuda_device, M):
    from binfer_b200.csrc import ops
    N, K = 300, 203
    a = torch.randn(130, K, device=cuda_device)
    w = torch.randn(N, K, device=cuda_device)
    out = torch.empty(M, N, device=cuda_device)
    ops.sgemm_nt(a[:M], w, out)
    ref = a[:M].double() @ w.double().T
    assert float((out.double() - ref).abs().max()) <= 2e-6 * float(ref.abs().max()) * math.sqrt(K)
    # a row's result does not depend on how many rows share the call (one order of summation)
    big = torch.empty(130, N, device=cuda_device)
    ops.sgemm_nt(a, w, big)
    assert torch.equal(out, big[:M])


# the three tile heights (16: few rows; 32, 64: by the tiles on the busiest SM), whole and ragged
@pytest.mark.parametrize("M,N,K", [(16, 64, 64), (17, 4100, 68), (32, 12288, 16), (65, 66, 132),
                                   (300, 8200, 80), (64, 64, 1)])
def test_sgemm_tiles_and_alignments_agree(cuda_device, M, N, K):
    from binfer_b200.csrc import ops
    a = torch.randn(M, K, device=cuda_device)
    w = torch.randn(N, K, device=cuda_device)
    out = torch.full((M, N), 7.0, device=cuda_device)
    ops.sgemm_nt(a, w, out)
    ref = a.double() @ w.double().T
    # runs of 64 terms: each rounding is at most half a unit of a partial sum
    bound = (64 + K / 64) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    assert bool(((out.double() - ref).abs() <= bound).all())
    # rows off the 16-byte boundaries are read term by term: the same sums
    off = torch.randn(M, K + 1, device=cuda_device)
    off[:, 1:] = a
    other = torch.full((M, N), 7.0, device=cuda_device)
    ops.sgemm_nt(off[:, 1:], w, other)
    assert torch.equal(out, other)
    one = torch.full((1, N), 7.0, device=cuda_device)
    ops.sgemm_nt(a[M - 1:], w, one)
    assert torch.equal(one[0], out[M - 1])


def test_sgemm_more_rows_than_a_grid_has_tiles(cuda_device):
    from binfer_b200.csrc import ops
    M = 64 * 65535 + 70
    a, w = torch.randn(M, 4, device=cuda_device), torch.randn(3, 4, device=cuda_device)
    out = torch.full((M, 3), 7.0, device=cuda_device)
    ops.sgemm_nt(a, w, out)
    bound = 5 * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)     # four products, their sums
    assert bool(((out.double() - a.double() @ w.double().T).abs() <= bound).all())


def _multiply_adds(a, w):
    from binfer_b200.csrc import ops
    out = torch.empty(a.shape[0], w.shape[0], device=a.device)
    ops.sgemm_nt(a, w, out, multiply_adds=True)
    return out


# 512 terms and more: three bfloat16 terms an operand.  Rows about the tiles (16, 112, 176), features
# about 128 and about the numbers of tiles that share K among 4, 2 and 1 CTAs; K about steps of 32
# and runs of 8 steps.
@pytest.mark.parametrize("M,N,K", [(1, 127, 512), (16, 129, 516), (17, 2304, 800), (112, 2305, 2048),
                                   (113, 64, 1027), (177, 9472, 640), (353, 9473, 544), (300, 8, 6145)])
def test_sgemm_of_terms(cuda_device, M, N, K):
    from binfer_b200.csrc import ops
    a = torch.randn(M, K, device=cuda_device)
    w = torch.randn(N, K, device=cuda_device)
    a[:, 1] *= 1e-30                                  # (terms far below the others)
    out = torch.full((M, N + 3), 7.0, device=cuda_device)[:, :N]
    ops.sgemm_nt(a, w, out)
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    # twelve products of terms a step, each sum cut off behind 24 bits (2^-23), then rounded sums
    # in runs of eight steps, of the runs, of four CTAs; products of terms left out, up to 2^-24
    bound = (12 * 2 + 8 + K / 256 + 4 + 1) * 2.0 ** -24 * size
    assert bool(((out.double() - ref).abs() <= bound).all())
    assert float((out.double() - ref).norm() / ref.norm()) < 1.6e-7      # (measured 1.1e-7)
    off = torch.randn(M, K + 1, device=cuda_device)
    off[:, 1:] = a
    other = torch.full((M, N), 7.0, device=cuda_device)
    ops.sgemm_nt(off[:, 1:], w, other)
    assert torch.equal(out, other)
    one = torch.full((1, N), 7.0, device=cuda_device)
    ops.sgemm_nt(a[M - 1:], w, one)
    assert torch.equal(one[0], out[M - 1])
    heads = torch.full((M, 2, N), 7.0, device=cuda_device)
    ops.sgemm_nt_batched(torch.stack([w[:1].expand(M, K), a], 1), torch.stack([w, w]), heads)
    assert torch.equal(heads[:, 1], out)
    assert int(ops.error_word(cuda_device).item()) == 0


@pytest.mark.parametrize("M,N,K,batch", [(1241, 130, 1024, 1), (300, 40, 600, 5), (40, 8, 2048, 7), (30, 300, 512, 9)])
def test_sgemm_of_terms_in_several_calls(cuda_device, monkeypatch, M, N, K, batch):
    """A product whose rows' terms pass the limit, cut by rows and by products: the same bits."""
    from binfer_b200.csrc import ops
    a = torch.randn(M, batch, K + 4, device=cuda_device)[:, :, :K]
    w = torch.randn(batch, N, K, device=cuda_device)
    outs = []
    for limit in (1 << 30, 6 * K * 1232, 6 * K * 300):
        monkeypatch.setattr(ops, "SGEMM_SPLIT_MAX_BYTES", limit)
        outs.append(torch.full((M, batch, N), 7.0, device=cuda_device))
        before = ops.launches()
        if batch == 1:
            ops.sgemm_nt(a[:, 0], w[0], outs[-1][:, 0])
        else:
            ops.sgemm_nt_batched(a, w, outs[-1])
        calls = ops._sgemm_split_calls(M, K, batch)
        assert ops.launches() - before == sum(1 + (m > 16) for _, _, _, m in calls)
    assert len(calls) > 1
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


# products side by side: each cluster size, tiles of 16 and of more rows
@pytest.mark.parametrize("batch,N,K", [(16, 128, 512), (9, 300, 520), (40, 512, 544)])
def test_sgemm_of_terms_many_products(cuda_device, batch, N, K):
    """Against float64 with test_sgemm_of_terms' bound; a row's bits alone and in company."""
    from binfer_b200.csrc import ops
    a = torch.randn(130, batch, K, device=cuda_device)
    w = torch.randn(batch, N, K, device=cuda_device)
    outs = []
    for M in (130, 16, 1):
        outs.append(torch.full((M, batch, N), 7.0, device=cuda_device))
        ops.sgemm_nt_batched(a[:M], w, outs[-1])
    ref, size = (torch.einsum("mbk,bnk->mbn", x, y) for x, y in (
        (a.double(), w.double()), (a.double().abs(), w.double().abs())))
    bound = (12 * 2 + 8 + K / 256 + 4 + 1) * 2.0 ** -24 * size
    assert bool(((outs[0].double() - ref).abs() <= bound).all())
    assert torch.equal(outs[1], outs[0][:16]) and torch.equal(outs[2], outs[0][:1])


# tiles of 16, 176 and 112 rows, features shared by clusters of 4 and 2 CTAs and not
@pytest.mark.parametrize("M,N,K", [(5, 300, 700), (40, 3000, 513), (200, 9500, 512), (224, 4200, 512)])
def test_sgemm_of_terms_with_products_that_overflow(cuda_device, M, N, K):
    """Finite operands whose products or sums leave float's range give the infinities and NaN of the
    multiply-adds; a smaller product of terms must not overflow with a sign of its own."""
    from binfer_b200.csrc import ops
    a, w = torch.randn(M, K, device=cuda_device), torch.randn(N, K, device=cuda_device)
    a[3, 7], w[5, 7], w[N - 1, 7] = 1.7e25, 1.3e20, -1.1e20
    a[2, 11], a[2, 12], w[8, 11], w[8, 12] = 1.7e25, -1.9e25, 1.1e20, 1.3e20
    a[M - 1], w[9] = 1e23 * torch.rand(K, device=cuda_device), 1e23 * torch.rand(K, device=cuda_device)
    a[1, 20], w[17, 20], a[1, 21], w[17, 21] = 1.5e19, 1.9e19, -1.4e19, 1.9e19     # (the sum is finite)
    out, want = torch.empty(M, N, device=cuda_device), _multiply_adds(a, w)
    ops.sgemm_nt(a, w, out)
    assert want[3, 5] == float("inf") and want[3, N - 1] == -float("inf") and not want[2, 8].isfinite()
    assert want[M - 1, 9] == float("inf") and want[1, 17].isfinite()
    assert torch.equal(out.isnan(), want.isnan())
    odd = ~want.isfinite() & ~want.isnan()
    assert torch.equal(out[odd], want[odd]) and bool(out[want.isfinite()].isfinite().all())
    size = a.double().abs() @ w.double().abs().T
    ref = a.double() @ w.double().T
    fin = want.isfinite()
    assert bool(((out.double() - ref).abs() <= 100 * 2.0 ** -24 * size)[fin].all())


@pytest.mark.parametrize("M,N,K", [(5, 300, 700), (40, 3000, 513), (200, 9500, 6145)])
def test_sgemm_of_terms_where_no_terms_are(cuda_device, M, N, K):
    """Rows without terms get the multiply-adds' sums, in their order: the same bits."""
    from binfer_b200.csrc import ops
    a, w = torch.randn(M, K, device=cuda_device), torch.randn(N, K, device=cuda_device)
    a[3, 9], w[:, 9], w[8, 5], a[:, 5] = 3.4e38, 0.0, -3.4e38, 0.0
    out, want = torch.empty(M, N, device=cuda_device), _multiply_adds(a, w)
    ops.sgemm_nt(a, w, out)
    assert bool(want.isfinite().all())
    assert torch.equal(out[3], want[3]) and torch.equal(out[:, 8], want[:, 8])


@pytest.mark.parametrize("M,N,K", [(5, 300, 700), (40, 3000, 513), (200, 9500, 512), (224, 4200, 800)])
def test_sgemm_of_terms_holds_floats_of_every_size(cuda_device, M, N, K):
    """Operands down to the smallest float keep all their bits, against large ones and among them;
    sums as large as float holds are there."""
    from binfer_b200.csrc import ops
    dev = cuda_device
    a, w = torch.randn(M, K, device=dev), torch.randn(N, K, device=dev)
    a *= 10.0 ** torch.tensor([0, -36, -38, -40, 6], device=dev)[torch.arange(M, device=dev) % 5][:, None]
    w *= 10.0 ** torch.tensor([30, 0, -36, 20], device=dev)[torch.arange(N, device=dev) % 4][:, None]
    a[0, 1::2] *= 1e-37                                      # in one row
    w[0, ::2] *= 1e-35
    out, want = torch.empty(M, N, device=dev), _multiply_adds(a, w)
    ops.sgemm_nt(a, w, out)
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    # (test_sgemm_of_terms' bound; each rounded result is off by half the smallest float at most)
    bound = (12 * 2 + 8 + K / 256 + 4 + 1) * 2.0 ** -24 * size + 2.0 ** -150
    assert bool(out.isfinite().all()) and bool(((out.double() - ref).abs() <= bound).all())
    for i in range(5):
        for j in range(4):
            r = ref[i::5, j::4]
            if float(r.abs().max()) > 1e-30:                 # (results that float itself holds)
                off = [float((x.double()[i::5, j::4] - r).norm() / r.norm()) for x in (out, want)]
                assert off[0] <= max(off[1], 1.6e-7), (i, j, off)


@pytest.mark.parametrize("M,N,K", [(5, 300, 700), (40, 3000, 513), (200, 9500, 512)])
def test_sgemm_of_terms_with_infinities(cuda_device, M, N, K):
    """Infinities, NaN and floats that no bfloat16 reaches give what multiply-adds give, and stay in
    their rows and columns."""
    from binfer_b200.csrc import ops
    a, w = torch.randn(M, K, device=cuda_device), torch.randn(N, K, device=cuda_device)
    clean = torch.empty(M, N, device=cuda_device)
    ops.sgemm_nt(a, w, clean)
    a[1, 5], a[2, 7], a[3, 9] = float("inf"), float("nan"), 3.4e38
    w[9, 2], w[11, 0], w[12, 5] = -float("inf"), float("nan"), 0.0
    w[:, 9] *= 1e-3
    a[:, 9][a[:, 9].abs() < 1e30] = 0.0
    want = (a.double() @ w.double().T).float()
    out = torch.empty(M, N, device=cuda_device)
    ops.sgemm_nt(a, w, out)
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.isinf(), want.isinf())
    fin = want.isfinite()
    # (rows of multiply-adds: one sequential sum)
    bound = K * 2.0 ** -24 * (torch.nan_to_num(a, 0, 0, 0).double().abs()
                              @ torch.nan_to_num(w, 0, 0, 0).double().abs().T)
    assert bool(((out.double() - want.double()).abs() <= bound)[fin].all())
    a[:, 9], w[:, 9] = 0.0, 0.0
    for t in (a, w):
        t[~t.isfinite().all(-1)] = 1.0
    again = torch.empty(M, N, device=cuda_device)
    ops.sgemm_nt(a, w, again)
    rows = torch.ones(M, dtype=torch.bool, device=cuda_device)
    rows[1:4] = False
    cols = torch.ones(N, dtype=torch.bool, device=cuda_device)
    cols[[9, 11]] = False
    assert torch.equal(out[rows][:, cols], again[rows][:, cols])


# ------------------------------------------------------- q/k norm, rotation, cache write
@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("nh,nkv,d,rot,norm", [(3, 1, 16, 16, True), (4, 2, 48, 24, True),
                                               (2, 2, 128, 128, False), (5, 5, 80, 0, True),
                                               (8, 2, 128, 128, True), (3, 1, 128, 64, True)])
def test_qk_norm_rope_kv_write(cuda_device, dtype, nh, nkv, d, rot, norm):
    from binfer_b200.csrc import ops
    T, ps, pages, eps, theta = 11, 4, 9, 1e-5, 5000.0
    dev = cuda_device
    qkv = torch.randn(T, (nh + 2 * nkv) * d, device=dev).to(dtype)
    qw = (1 + 0.1 * torch.randn(d, device=dev)) if norm else None
    kw = (1 + 0.1 * torch.randn(d, device=dev)) if norm else None
    pos = torch.tensor([0, 1, 2, 3, 40, 41, 1000, 7, 8, 9, 10], dtype=torch.int32, device=dev)
    slots = torch.randperm(pages * ps)[:T].to(torch.int32).to(dev)
    slots[3] = -1                                   # this token is not written
    inv = None
    if rot:
        i = torch.arange(rot // 2, dtype=torch.float64)
        inv = (theta ** (-2.0 * i / rot)).float().to(dev)
    kc = torch.zeros(pages, nkv, ps, d, device=dev, dtype=dtype)
    vc = torch.zeros_like(kc)
    q_out = torch.empty(T, nh * d, device=dev, dtype=dtype)
    err = _err(dev)
    ops.qk_norm_rope_kv_write(qkv, qw, kw, inv, pos, slots, q_out, kc, vc, nh, nkv, d, eps, err)
    assert int(err.item()) == 0
    x = qkv.double().cpu()
    q = x[:, :nh * d].view(T, nh, d)
    k = x[:, nh * d:(nh + nkv) * d].view(T, nkv, d)
    v = x[:, (nh + nkv) * d:].view(T, nkv, d)
    if norm:
        q, k = P.rms_norm(q, qw.double().cpu(), eps), P.rms_norm(k, kw.double().cpu(), eps)
    if rot:
        ang = P.rope_angles(pos.cpu(), rot, theta)
        q, k = P.apply_rope(q, ang), P.apply_rope(k, ang)
    _close(q_out.view(T, nh, d), q, dtype)
    for t in range(T):
        s = int(slots[t])
        if s < 0:
            continue
        _close(kc[s // ps, :, s % ps], k[t], dtype)
        _close(vc[s // ps, :, s % ps], v[t], dtype)
    assert float(kc.abs().sum(dim=(1, 3)).flatten().count_nonzero()) == T - 1


@pytest.mark.parametrize("nh,nkv,norm", [(8, 2, True), (32, 8, True), (5, 1, True), (64, 8, True),
                                         (3, 3, False)])
def test_qk_norm_rope_kv_write_many_tokens(cuda_device, nh, nkv, norm):
    """Heads of 128 and more than 64 tokens: a block per token whose warps walk the heads, six
    of them asked for at a time.  Odd head counts, 80 heads; some tokens are not written;
    positions are far apart."""
    from binfer_b200.csrc import ops
    T, d, ps, eps, theta = 203, 128, 16, 1e-6, 1e6
    dev = cuda_device
    g = torch.Generator().manual_seed(nh)
    qkv = torch.randn(T, (nh + 2 * nkv) * d, generator=g).to(BF16).to(dev)
    qw = (1 + 0.1 * torch.randn(d, generator=g)).to(dev) if norm else None
    kw = (1 + 0.1 * torch.randn(d, generator=g)).to(dev) if norm else None
    pos = (torch.arange(T) * 37 % 5000).to(torch.int32).to(dev)
    pages = T // ps + 3
    slots = torch.randperm(pages * ps, generator=g)[:T].to(torch.int32)
    slots[7] = slots[100] = -1
    slots = slots.to(dev)
    i = torch.arange(d // 2, dtype=torch.float64)
    inv = (theta ** (-2.0 * i / d)).float().to(dev)
    kc = torch.zeros(pages, nkv, ps, d, device=dev, dtype=BF16)
    vc = torch.zeros_like(kc)
    q_out = torch.empty(T, nh * d, device=dev, dtype=BF16)
    err = _err(dev)
    ops.qk_norm_rope_kv_write(qkv, qw, kw, inv, pos, slots, q_out, kc, vc, nh, nkv, d, eps, err)
    assert int(err.item()) == 0
    x = qkv.double().cpu()
    q = x[:, :nh * d].view(T, nh, d)
    k = x[:, nh * d:(nh + nkv) * d].view(T, nkv, d)
    v = x[:, (nh + nkv) * d:].view(T, nkv, d)
    if norm:
        q, k = P.rms_norm(q, qw.double().cpu(), eps), P.rms_norm(k, kw.double().cpu(), eps)
    ang = P.rope_angles(pos.cpu(), d, theta)
    q, k = P.apply_rope(q, ang), P.apply_rope(k, ang)
    _close(q_out.view(T, nh, d), q, BF16)
    sl = slots.cpu()
    live = sl >= 0
    got_k = kc.cpu()[sl[live] // ps, :, sl[live] % ps]
    got_v = vc.cpu()[sl[live] // ps, :, sl[live] % ps]
    _close(got_k, k[live], BF16)
    _close(got_v, v[live], BF16)
    assert int(kc.abs().sum(dim=(1, 3)).flatten().count_nonzero()) == int(live.sum())


# ----------------------------------------------------------------------- attention
def _paged(k, v, ps, dev, dtype, seed=0, neighbours=False):
    """Scatter dense k, v ``[n, nkv, d]`` of one request into shuffled pages (or, with
    ``neighbours``, into pages that lie side by side in the pool).
    Returns caches ``[pages, nkv, ps, d]`` and the block table."""
    n, nkv, d = k.shape
    n_pages = -(-n // ps)
    total = n_pages + 5
    g = torch.Generator().manual_seed(seed)
    ids = (torch.randperm(total - 1, generator=g)[:n_pages] + 1).tolist()   # page 0 unused
    if neighbours:
        ids = list(range(3, 3 + n_pages))
    kc = torch.randn(total, nkv, ps, d, generator=g).to(dtype)              # junk elsewhere
    vc = torch.randn(total, nkv, ps, d, generator=g).to(dtype)
    for j in range(n):
        kc[ids[j // ps], :, j % ps] = k[j].to(dtype)
        vc[ids[j // ps], :, j % ps] = v[j].to(dtype)
    return kc.to(dev), vc.to(dev), ids


def _attention_case(dev, dtype, nh, nkv, d, ps, ctxs, qlens, window, spike=False, seed=0,
                    neighbours=False):
    """Requests with contexts ``ctxs``, the last ``qlens`` tokens of each being queries."""
    g = torch.Generator().manual_seed(seed)
    ks, vs, qs, tables, refs = [], [], [], [], []
    kcs, vcs = [], []
    page_base = 0
    for b, (n, ql) in enumerate(zip(ctxs, qlens)):
        k = torch.randn(n, nkv, d, generator=g).to(dtype).double()
        v = torch.randn(n, nkv, d, generator=g).to(dtype).double()
        q = torch.randn(n, nh, d, generator=g).to(dtype).double()
        if spike and n > 40:
            # one far key stands out: its score beats hundreds of others.  With a window it
            # is the first key inside the last query's window, and the key just outside
            # stands out even more, so reading one key too many shows as well.
            far = 3 if window is None else max(0, n - window)
            k[far] = 0
            k[far, :, 0] = 32.0
            q[-1, :, 0] = 16.0
            v[far] = 5.0
            if window is not None and far > 0:
                k[far - 1] = 0
                k[far - 1, :, 0] = 64.0
                v[far - 1] = -7.0
        ref = P.causal_attention(q, k, v, d ** -0.5, window)[n - ql:]
        kc, vc, ids = _paged(k, v, ps, "cpu", dtype, seed + b, neighbours)
        kcs.append(kc)
        vcs.append(vc)
        tables.append([i + page_base for i in ids])
        page_base += kc.shape[0]
        qs.append(q[n - ql:])
        refs.append(ref)
    width = max(len(t) for t in tables)
    bt = torch.zeros(len(ctxs), width, dtype=torch.int32)
    for b, t in enumerate(tables):
        bt[b, :len(t)] = torch.tensor(t, dtype=torch.int32)
    q_all = torch.cat(qs).to(dtype).reshape(-1, nh * d).to(dev)
    pos = torch.cat([torch.arange(n - ql, n) for n, ql in zip(ctxs, qlens)]).to(torch.int32).to(dev)
    sot = torch.cat([torch.full((ql,), b) for b, ql in enumerate(qlens)]).to(torch.int32).to(dev)
    return (q_all, torch.cat(kcs).to(dev), torch.cat(vcs).to(dev), sot, pos, bt.to(dev),
            torch.cat(refs).reshape(-1, nh * d))


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("nh,nkv,d,ps,window,spike", [
    (4, 2, 16, 16, None, False), (6, 1, 32, 8, None, True), (5, 5, 48, 4, 24, True),
    (8, 2, 128, 16, None, True), (3, 3, 80, 5, 33, False), (2, 1, 256, 16, 100, True)])
def test_paged_attention_generic(cuda_device, dtype, nh, nkv, d, ps, window, spike):
    from binfer_b200.csrc import ops
    ctxs, qlens = [70, 1, 129, 300], [70, 1, 5, 2]
    q, kc, vc, sot, pos, bt, ref = _attention_case(cuda_device, dtype, nh, nkv, d, ps, ctxs,
                                                   qlens, window, spike)
    out = torch.empty_like(q)
    err = _err(cuda_device)
    ops.paged_attention_generic(q, kc, vc, sot, pos, bt, out, nh, nkv, d, window, d ** -0.5, err)
    assert int(err.item()) == 0
    _close(out, ref, dtype)


@pytest.mark.parametrize("nh,nkv,d,ps,window,spike", [
    (4, 2, 32, 16, None, False), (6, 1, 32, 8, None, True), (8, 2, 128, 16, None, True),
    (32, 8, 128, 16, None, False), (5, 5, 96, 4, 24, True), (3, 3, 64, 5, 200, True),
    (2, 1, 256, 16, 100, True), (20, 1, 64, 16, None, True), (4, 4, 128, 64, 130, True)])
@pytest.mark.parametrize("variant", ["cp_async", "tma", "persistent"])
def test_decode_attention_split_kv(cuda_device, nh, nkv, d, ps, window, spike, variant):
    """Contexts on both sides of the 128-key split edge, and long ones; every way of
    fetching the tiles."""
    from binfer_b200.csrc import ops
    if variant != "cp_async" and not (d in (64, 128, 256) and ps >= 8 and 128 % ps == 0):
        pytest.skip(f"the {variant} variant does not take this head or page size")
    if variant == "persistent" and nh // nkv > 16:
        pytest.skip("the persistent variant takes at most 16 heads per kv head")
    ctxs = [1, 127, 128, 129, 300, 1000, 45]
    qlens = [1] * len(ctxs)
    q, kc, vc, sot, pos, bt, ref = _attention_case(cuda_device, BF16, nh, nkv, d, ps, ctxs,
                                                   qlens, window, spike, seed=3)
    out = torch.zeros_like(q)
    err = _err(cuda_device)
    ops.decode_attention(q, kc, vc, None, len(ctxs), sot, pos, bt, out, nh, nkv, d, window,
                         d ** -0.5, max(ctxs) + 500, err, variant=variant)
    assert int(err.item()) == 0
    _close(out, ref, BF16)
    # a subset of rows, given by index, gives the same bits for those rows
    rows = torch.tensor([5, 2, 4], dtype=torch.int32, device=cuda_device)
    out2 = torch.zeros_like(q)
    ops.decode_attention(q, kc, vc, rows, 3, sot, pos, bt, out2, nh, nkv, d, window,
                         d ** -0.5, max(ctxs), err, variant=variant)
    for r in (5, 2, 4):
        assert torch.equal(out2[r], out[r])
    assert float(out2[0].abs().max()) == 0.0


@pytest.mark.parametrize("nh,nkv,d,ps,cap", [(8, 2, 128, 16, 3.0), (6, 3, 64, 8, 0.7),
                                              (4, 4, 256, 32, 5.0), (16, 8, 128, 64, 0.0)])
def test_decode_attention_soft_cap_into_a_column_block(cuda_device, nh, nkv, d, ps, cap):
    """The persistent variant with scores through ``c tanh(s / c)``, the result times a factor
    and written into a column block of a wider buffer whose other columns stay as they were.
    The scores are large (a scale of one on long vectors), so a cap left out would show."""
    from binfer_b200.csrc import ops
    dev, gen = cuda_device, torch.Generator().manual_seed(nh * 100 + d)
    ctxs, scale, factor, left, right = [1, 127, 129, 300, 700, 45], 0.5, 1.3, 8, 24
    kcs, vcs, tables, qs, refs, base = [], [], [], [], [], 0
    for b, n in enumerate(ctxs):
        k = torch.randn(n, nkv, d, generator=gen).to(BF16).double()
        v = torch.randn(n, nkv, d, generator=gen).to(BF16).double()
        q = torch.randn(nh, d, generator=gen).to(BF16).double()
        kh = k.repeat_interleave(nh // nkv, dim=1)
        vh = v.repeat_interleave(nh // nkv, dim=1)
        sc = torch.einsum("hd,nhd->hn", q, kh) * scale
        if cap > 0:
            sc = cap * torch.tanh(sc / cap)
        refs.append(factor * torch.einsum("hn,nhd->hd", torch.softmax(sc, dim=-1), vh))
        kc, vc, ids = _paged(k, v, ps, "cpu", BF16, 50 + b, False)
        kcs.append(kc)
        vcs.append(vc)
        tables.append([i + base for i in ids])
        base += kc.shape[0]
        qs.append(q)
    bt = torch.zeros(len(ctxs), max(len(t) for t in tables), dtype=torch.int32)
    for b, t in enumerate(tables):
        bt[b, :len(t)] = torch.tensor(t, dtype=torch.int32)
    q_all = torch.stack(qs).to(BF16).reshape(len(ctxs), nh * d).to(dev)
    pos = torch.tensor([n - 1 for n in ctxs], dtype=torch.int32, device=dev)
    sot = torch.arange(len(ctxs), dtype=torch.int32, device=dev)
    wide = torch.full((len(ctxs), left + nh * d + right), 7.0, dtype=BF16, device=dev)
    out = wide[:, left:left + nh * d]
    kc, vc = torch.cat(kcs).to(dev), torch.cat(vcs).to(dev)
    assert ops.decode_attention_takes_capped(q_all, kc, nh, nkv, d, d, len(ctxs))
    err = _err(dev)
    ops.decode_attention(q_all, kc, vc, None, len(ctxs), sot, pos, bt.to(dev), out, nh, nkv, d,
                         None, scale, max(ctxs) + 300, err, variant="persistent", softcap=cap,
                         out_scale=factor)
    assert int(err.item()) == 0
    _close(out, torch.stack(refs).reshape(len(ctxs), nh * d), BF16)
    assert bool((wide[:, :left] == 7.0).all()) and bool((wide[:, left + nh * d:] == 7.0).all())
    if cap > 0:
        plain = torch.empty((len(ctxs), nh * d), dtype=BF16, device=dev)
        ops.decode_attention(q_all, kc, vc, None, len(ctxs), sot, pos, bt.to(dev), plain, nh, nkv,
                             d, None, scale, max(ctxs) + 300, err, variant="persistent")
        assert float((plain.float() * factor - out.float()).abs().max()) > 0.05


@pytest.mark.parametrize("nh,nkv,d,ps,window", [
    (8, 2, 128, 16, None), (32, 8, 128, 16, 300), (6, 3, 64, 8, None), (4, 4, 256, 32, None),
    (8, 4, 128, 64, 1000)])
def test_decode_attention_with_pages_side_by_side(cuda_device, nh, nkv, d, ps, window):
    """Tiles whose pages are neighbours in the pool arrive as one box: the same bits as with
    the pages scattered (one box a page), and the plain result.  Contexts that end inside a
    tile, rows shorter than a tile, a window that starts inside one."""
    from binfer_b200.csrc import ops
    ctxs = [1, 127, 128, 129, 300, 1000, 45, 2050, 640]
    qlens = [1] * len(ctxs)
    outs = []
    for neighbours in (True, False):
        q, kc, vc, sot, pos, bt, ref = _attention_case(
            cuda_device, BF16, nh, nkv, d, ps, ctxs, qlens, window, True, seed=13,
            neighbours=neighbours)
        out = torch.zeros_like(q)
        err = _err(cuda_device)
        ops.decode_attention(q, kc, vc, None, len(ctxs), sot, pos, bt, out, nh, nkv, d, window,
                             d ** -0.5, max(ctxs), err, variant="persistent")
        assert int(err.item()) == 0
        _close(out, ref, BF16)
        outs.append(out)
    assert torch.equal(outs[0], outs[1]), "the result depends on where the pages lie"


@pytest.mark.parametrize("nh,nkv,d,ps,window", [
    (8, 4, 128, 16, None), (12, 4, 64, 32, 700), (4, 2, 256, 8, None), (16, 1, 128, 128, None)])
def test_decode_attention_persistent_ring_wraps(cuda_device, nh, nkv, d, ps, window):
    """So many (row, kv head, split) items that every resident CTA takes more of them than its
    ring of tile slots holds, with rows of very different lengths; compared with the plain
    result and, bit for bit, with the one-CTA-per-split kernel's partial sums merged the
    same way."""
    from binfer_b200.csrc import ops
    ctxs = [2900, 1, 1500, 130, 3001, 777, 2048, 64, 2500, 3, 1999, 2300] * 2
    qlens = [1] * len(ctxs)
    q, kc, vc, sot, pos, bt, ref = _attention_case(cuda_device, BF16, nh, nkv, d, ps, ctxs,
                                                   qlens, window, True, seed=11)
    err = _err(cuda_device)
    out = torch.zeros_like(q)
    ops.decode_attention(q, kc, vc, None, len(ctxs), sot, pos, bt, out, nh, nkv, d, window,
                         d ** -0.5, max(ctxs), err, variant="persistent")
    assert int(err.item()) == 0
    _close(out, ref, BF16)
    again = torch.zeros_like(q)
    ops.decode_attention(q, kc, vc, None, len(ctxs), sot, pos, bt, again, nh, nkv, d, window,
                         d ** -0.5, max(ctxs), err, variant="persistent")
    assert torch.equal(out, again), "the result depends on timing"


@pytest.mark.parametrize("window", [None, 5000])
@pytest.mark.parametrize("variant", ["cp_async", "tma", "persistent"])
def test_decode_attention_more_splits_than_one_merge_pass(cuda_device, variant, window):
    """Contexts beyond 16384 keys: the merge kernel's shape for many splits, more of them than
    a lane asks for at once, and (with a window) a first split that is not split 0.  One key
    far back is made to stand out, so a lost pass would show."""
    from binfer_b200.csrc import ops
    nh, nkv, d, ps = 4, 2, 64, 64
    ctxs, qlens = [20000, 16385, 300], [1, 1, 1]
    q, kc, vc, sot, pos, bt, ref = _attention_case(cuda_device, BF16, nh, nkv, d, ps, ctxs,
                                                   qlens, window, True, seed=5)
    out = torch.zeros_like(q)
    err = _err(cuda_device)
    ops.decode_attention(q, kc, vc, None, len(ctxs), sot, pos, bt, out, nh, nkv, d, window,
                         d ** -0.5, max(ctxs), err, variant=variant)
    assert int(err.item()) == 0
    _close(out, ref, BF16)


@pytest.mark.parametrize("variant", ["cp_async", "tma", "persistent"])
def test_decode_attention_flags_a_row_beyond_its_scratch(cuda_device, variant):
    """Scratch with room for one split and a row of 200 keys, which needs two: the error
    word's bit says so, nothing behind the scratch is touched, and the row that fits is
    right all the same."""
    from binfer_b200.csrc import ops
    nh, nkv, d, ps = 8, 2, 128, 16
    ctxs = [200, 90]
    q, kc, vc, sot, pos, bt, ref = _attention_case(cuda_device, BF16, nh, nkv, d, ps, ctxs,
                                                   [1, 1], None, seed=21)
    cells = len(ctxs) * nh * 1
    buf = torch.full((cells * (d + 2) + 8192,), 777.0, dtype=torch.float32, device=cuda_device)
    part_o = buf[:cells * d].view(len(ctxs), nh, 1, d)
    part_ml = buf[cells * d:cells * (d + 2)].view(len(ctxs), nh, 1, 2)
    out = torch.zeros_like(q)
    err = _err(cuda_device)
    ops.decode_attention(q, kc, vc, None, len(ctxs), sot, pos, bt, out, nh, nkv, d, None,
                         d ** -0.5, max(ctxs), err, variant=variant, scratch=(part_o, part_ml))
    torch.cuda.synchronize()
    assert int(err.item()) == 16
    err.zero_()
    assert bool((buf[cells * (d + 2):] == 777.0).all()), "memory behind the scratch was written"
    _close(out[1], ref[1], BF16)
    assert bool(torch.isfinite(out.float()).all())


@pytest.mark.parametrize("M,N,K,bn,c", [(8, 4096, 4096, 128, 4), (3, 200, 512, 64, 2),
                                        (16, 1000, 320, 80, 1), (64, 4096, 4096, 128, 4),
                                        (37, 1024, 2048, 64, 4), (27, 520, 1024, 64, 2),
                                        (32, 4096, 4096, 128, 4)])
def test_gemm_cluster_adds_into_the_stream_and_prepares_the_norm(cuda_device, M, N, K, bn, c):
    """resid += x w^T in float; xt = bf16(resid * norm_w); the partial sums of squares add up
    to the rows' sums, so that xt times the factor is the RMSNorm of the new stream."""
    from binfer_b200.csrc import ops
    g = torch.Generator().manual_seed(N + K)
    x = torch.randn(M, K, generator=g).to(BF16).to(cuda_device)
    w = (0.05 * torch.randn(N, K, generator=g)).to(BF16).to(cuda_device)
    resid0 = (3.0 * torch.randn(M, N, generator=g)).to(cuda_device)
    nw = (1.0 + 0.1 * torch.randn(N, generator=g)).to(cuda_device)
    eps = 1e-5
    resid = resid0.clone()
    err = ops.error_word(cuda_device)
    got = ops.gemm_bf16_cluster_add_norm(x, w, resid, nw, eps, err, bn, c)
    assert got is not None and int(err.item()) == 0
    xt, scale = got
    want = resid0.double().cpu() + x.double().cpu() @ w.double().cpu().T
    assert float((resid.double().cpu() - want).abs().max()) <= 4e-7 * math.sqrt(K) * float(want.abs().max())
    assert scale.partials.shape == (M, -(-N // bn) * c) and scale.width == N
    ss = scale.partials.double().sum(1).cpu()
    assert torch.allclose(ss, (want ** 2).sum(1), rtol=1e-5)
    normed = want * torch.rsqrt((want ** 2).mean(1, keepdim=True) + eps) * nw.double().cpu()
    _close(xt.float() * scale.factors().unsqueeze(1), normed, BF16)
    # the factor applied by the kernels that come after the next product
    I = 264
    gu = torch.randn(M, 2 * I, generator=g).to(BF16).to(cuda_device)
    out = torch.empty(M, I, device=cuda_device, dtype=BF16)
    ops.silu_mul(gu, out, row_scale=scale)
    f = scale.factors().double().cpu().unsqueeze(1)
    gd = gu.double().cpu() * f
    _close(out, gd[:, :I] / (1 + torch.exp(-gd[:, :I])) * gd[:, I:], BF16)


@pytest.mark.parametrize("T,nh,nkv,d,rot,K,bn,c,norm,scaled", [
    (8, 32, 8, 128, 128, 4096, 128, 2, True, True),      # the 8B decode step's arrangement
    (5, 6, 2, 64, 64, 1024, 128, 2, True, False),        # two heads a tile
    (13, 5, 1, 96, 64, 1280, 192, 4, True, True),        # a rotation over part of the head
    (16, 3, 3, 256, 256, 512, 256, 1, False, False),     # one CTA a tile, no head norms
    (37, 7, 1, 128, 0, 2304, 128, 5, True, True),        # token rows beyond 32, no rotation
    (21, 4, 2, 64, 64, 1024, 128, 2, True, True),        # 17 to 32 token rows
    (2, 4, 0, 128, 128, 640, 256, 2, True, False),       # queries only: another layer's pages
    (1, 8, 2, 32, 0, 768, 32, 3, False, True),           # fewer tokens than CTAs in a cluster
])
def test_gemm_cluster_qkv_norms_turns_and_stores(cuda_device, T, nh, nkv, d, rot, K, bn, c, norm,
                                                 scaled):
    """The q/k/v projection with its epilogue against the product followed by the plain
    head norm, rotation and store: q, and every page slot of k and v (untouched slots
    stay zero, a token with a negative slot is not stored)."""
    from binfer_b200.csrc import ops
    dev, ps, eps, theta = cuda_device, 4, 1e-5, 5000.0
    pages = -(-T // ps) + 3
    g = torch.Generator().manual_seed(T * 1000 + K)
    x = torch.randn(T, K, generator=g).to(BF16).to(dev)
    w = (torch.randn((nh + 2 * nkv) * d, K, generator=g) / math.sqrt(K)).to(BF16).to(dev)
    qw = (1 + 0.1 * torch.randn(d, generator=g)).to(dev) if norm else None
    kw = (1 + 0.1 * torch.randn(d, generator=g)).to(dev) if norm else None
    pos = torch.randint(0, 3000, (T,), generator=g).to(torch.int32).to(dev)
    slots = torch.randperm(pages * ps, generator=g)[:T].to(torch.int32).to(dev)
    if T > 3:
        slots[3] = -1
    inv = None
    if rot:
        i = torch.arange(rot // 2, dtype=torch.float64)
        inv = (theta ** (-2.0 * i / rot)).float().to(dev)
    scale = None
    factor = torch.ones(T, dtype=torch.float64)
    if scaled:
        partials = (torch.rand(T, 37, generator=g) * 40).to(dev)
        scale = ops.RowScale(partials, 1536, 1e-6)
        factor = scale.factors().double().cpu()
    kc = torch.zeros(pages, max(nkv, 1), ps, d, device=dev, dtype=BF16) if nkv else None
    vc = torch.zeros_like(kc) if nkv else None
    q_out = torch.empty(T, nh * d, device=dev, dtype=BF16)
    err = _err(dev)
    assert ops.gemm_bf16_cluster_qkv(x, w, qw, kw, inv, pos, slots if nkv else None, q_out, kc, vc,
                                     nh, nkv, d, eps, err, bn, c, row_scale=scale)
    assert int(err.item()) == 0
    y = (x.double().cpu() @ w.double().cpu().T) * factor[:, None]
    q = y[:, :nh * d].view(T, nh, d)
    k = y[:, nh * d:(nh + nkv) * d].view(T, nkv, d)
    v = y[:, (nh + nkv) * d:].view(T, nkv, d)
    if norm:
        q = P.rms_norm(q, qw.double().cpu(), eps)
        k = P.rms_norm(k, kw.double().cpu(), eps) if nkv else k
    if rot:
        ang = P.rope_angles(pos.cpu(), rot, theta)
        q = P.apply_rope(q, ang)
        k = P.apply_rope(k, ang) if nkv else k
    _close(q_out.view(T, nh, d), q, BF16)
    if not nkv:
        return
    stored = 0
    for t in range(T):
        s_ = int(slots[t])
        if s_ < 0:
            continue
        stored += 1
        _close(kc[s_ // ps, :, s_ % ps], k[t], BF16)
        _close(vc[s_ // ps, :, s_ % ps], v[t], BF16)
    assert int(kc.abs().sum(dim=(1, 3)).flatten().count_nonzero()) == stored
    assert int(vc.abs().sum(dim=(1, 3)).flatten().count_nonzero()) == stored


def test_gemm_cluster_qkv_plan_keeps_whole_heads(cuda_device):
    from binfer_b200.csrc import ops
    sms = ops.num_sms(cuda_device)
    for features, K, d in [(6144, 4096, 128), (2560, 1536, 128), (10240, 5120, 128),
                           (1536, 1024, 64), (1280, 2048, 256), (480, 640, 96)]:
        plan = ops.gemm_cluster_qkv_plan(features, K, d, cuda_device)
        assert plan is not None, (features, K, d)
        bn, c, ctas = plan
        assert bn % d == 0 and bn <= 256 and 1 <= c <= 8 and (K // 64) // c >= 4
        assert ctas == -(-features // bn) * c <= sms
    assert ops.gemm_cluster_qkv_plan(4096, 4096, 80, cuda_device) is None     # not whole warps


@pytest.mark.parametrize("T,I,K,bn,scaled", [
    (8, 12288, 4096, 0, True),        # the 8B decode step's shape, the plan's tile
    (5, 1000, 512, 0, False),         # outputs that are no multiple of the tile
    (16, 2504, 320, 48, True),        # 24 outputs a tile: the last chunk of a tile is cut
    (37, 264, 1024, 256, True),       # token rows beyond 32; one tile holds part of the outputs
    (29, 1000, 512, 0, True),         # 17 to 32 token rows: 64-row products, two lane quarters
    (1, 4480, 1536, 112, False),
])
def test_gemm_swiglu_matches_product_then_activation(cuda_device, T, I, K, bn, scaled):
    """silu(f g) * (f u) of the stacked gate/up product, straight from tensor memory."""
    from binfer_b200.csrc import ops
    dev = cuda_device
    g = torch.Generator().manual_seed(I + K + T)
    x = torch.randn(T, K, generator=g).to(BF16).to(dev)
    w = (2.0 * torch.randn(2 * I, K, generator=g) / math.sqrt(K)).to(BF16).to(dev)
    scale, f = None, torch.ones(T, dtype=torch.float64)
    if scaled:
        scale = ops.RowScale((torch.rand(T, 130, generator=g) * 8).to(dev), 512, 1e-6)
        f = scale.factors().double().cpu()
    if bn == 0:
        bn, ctas = ops.gemm_swiglu_plan(I, K, dev)
        assert bn % 16 == 0 and ctas == -(-I // (bn // 2)) <= ops.num_sms(dev)
    out = torch.full((T, I), 7.0, device=dev, dtype=BF16)
    err = _err(dev)
    assert ops.gemm_bf16_swiglu(x, w, out, err, bn, row_scale=scale)
    assert int(err.item()) == 0
    y = (x.double().cpu() @ w.double().cpu().T) * f[:, None]
    gate, up = y[:, :I], y[:, I:]
    _close(out, gate / (1 + torch.exp(-gate)) * up, BF16)


# ------------------------------------------------------------------------ sampling
def _sample(dev, logits, temperature, top_k=0, top_p=1.0, u=0.0):
    from binfer_b200.csrc import ops
    R = logits.shape[0]
    f = lambda v, dt: torch.full((R,), v, dtype=dt, device=dev)
    uu = torch.as_tensor(u, dtype=torch.float32, device=dev).expand(R).contiguous()
    out = torch.empty(R, dtype=torch.int32, device=dev)
    ops.sample(logits, f(temperature, torch.float32), f(top_k, torch.int32),
               f(top_p, torch.float32), uu, out)
    return out.cpu().tolist()


def test_argmax_lowest_index_on_ties(cuda_device):
    logits = torch.randn(5, 3001, device=cuda_device)
    logits[0, [7, 2000, 2999]] = 50.0
    logits[1, 3000] = 50.0
    logits[2, 0] = 50.0
    logits[3] = 1.0                                   # all equal
    got = _sample(cuda_device, logits, 0.0)
    assert got[:4] == [7, 3000, 0, 0]
    assert got[4] == int(torch.argmax(logits[4]))


@pytest.mark.parametrize("temperature,top_k,top_p", [(0.8, 0, 1.0), (1.3, 5, 1.0), (0.7, 0, 0.6),
                                                     (1.0, 40, 0.9), (2.0, 1, 1.0)])
def test_sampling_matches_plain_sampler(cuda_device, temperature, top_k, top_p):
    g = torch.Generator().manual_seed(5)
    V = 1237
    logits = (3 * torch.randn(24, V, generator=g))
    us = torch.rand(24, generator=g)
    got = _sample(cuda_device, logits.to(cuda_device), temperature, top_k, top_p, us)
    for r in range(24):
        want = P.sample(logits[r], temperature, top_k, top_p, uniform=float(us[r]))
        if got[r] != want:
            # only a draw that lands within float rounding of a boundary may differ
            s = logits[r].double() / temperature
            p = torch.softmax(s, 0)
            cum = torch.cumsum(p, 0)
            assert abs(float(cum[min(got[r], want)]) - float(us[r])) < 1e-4, (r, got[r], want)


def test_top_k_confines_support_and_penalty(cuda_device):
    from binfer_b200.csrc import ops
    g = torch.Generator().manual_seed(1)
    logits = torch.randn(1, 500, generator=g)
    top = set(torch.topk(logits[0], 5).indices.tolist())
    dev_logits = logits.to(cuda_device).repeat(64, 1).contiguous()
    got = _sample(cuda_device, dev_logits, 1.5, top_k=5, u=torch.rand(64, generator=g))
    assert set(got) <= top and len(set(got)) > 1
    # repetition penalty flips the argmax (s > 0 ? s / pen : s * pen), twice for two occurrences
    lg = torch.tensor([[1.0, 3.0, 2.9, -1.0]], device=cuda_device)
    items = torch.tensor([[0, 1, 2], [0, 3, 1]], dtype=torch.int32, device=cuda_device)
    ops.repetition_penalty(lg, items, torch.tensor([1.5], device=cuda_device))
    assert torch.allclose(lg.cpu(), torch.tensor([[1.0, 3.0 / 2.25, 2.9, -1.5]]))
    assert _sample(cuda_device, lg, 0.0) == [2]


# ------------------------------------------------------------- tcgen05 matrix product
@pytest.mark.parametrize("M,N,K", [(1, 300, 200), (8, 128, 64), (7, 6144, 4096), (16, 4096, 4104),
                                   (33, 1000, 512), (64, 4096, 12288), (65, 272, 72),
                                   (128, 256, 64), (200, 700, 1000), (513, 2100, 2048)])
@pytest.mark.parametrize("out_dtype", [BF16, F32])
def test_gemm_bf16_tcgen05(cuda_device, M, N, K, out_dtype):
    """Token counts on both sides of the 128-row tile, widths and depths that are no
    multiple of the tile, bfloat16 and float32 results."""
    from binfer_b200.csrc import ops
    g = torch.Generator().manual_seed(M * 7 + N)
    x = torch.randn(M, K, generator=g).to(BF16).to(cuda_device)
    w = (0.05 * torch.randn(N, K, generator=g)).to(BF16).to(cuda_device)
    out = torch.full((M, N), 99.0, device=cuda_device, dtype=out_dtype)
    err = ops.error_word(cuda_device)
    assert ops.gemm_bf16(x, w, out, err)
    assert int(err.item()) == 0
    ref = x.double().cpu() @ w.double().cpu().T
    if out_dtype == BF16:
        _close(out, ref, BF16)
    else:
        # float accumulation of K products in the tensor core: error grows like sqrt(K)
        err_rel = float((out.double().cpu() - ref).abs().max() / ref.abs().max())
        assert err_rel <= 4e-7 * math.sqrt(K), err_rel
    # every tile width gives the same sums (one order of accumulation over K)
    for bn in (16, 48, 256):
        other = torch.empty_like(out)
        assert ops.gemm_bf16(x, w, other, err, bn=bn)
        assert torch.equal(other, out), f"tile width {bn} changes the result"


@pytest.mark.parametrize("M,N,K", [(1, 300, 200), (130, 128, 64), (256, 6144, 4096),
                                   (300, 1000, 520), (513, 2100, 2048), (700, 272, 72),
                                   (2048, 4096, 1024), (1000, 40, 4104)])
@pytest.mark.parametrize("out_dtype", [BF16, F32])
def test_gemm_bf16_pair(cuda_device, M, N, K, out_dtype):
    """The product on pairs of SMs: token counts on both sides of the 256-row tile and of a
    CTA's 128 rows, widths and depths that are no multiple of the tile, more tiles than pairs
    (the rings of stages and the two accumulators wrap), bfloat16 and float32 results."""
    from binfer_b200.csrc import ops
    g = torch.Generator().manual_seed(M * 7 + N)
    x = torch.randn(M, K, generator=g).to(BF16).to(cuda_device)
    w = (0.05 * torch.randn(N, K, generator=g)).to(BF16).to(cuda_device)
    out = torch.full((M, N), 99.0, device=cuda_device, dtype=out_dtype)
    err = ops.error_word(cuda_device)
    assert ops.gemm_bf16_pair(x, w, out, err)
    assert int(err.item()) == 0
    ref = x.double().cpu() @ w.double().cpu().T
    if out_dtype == BF16:
        _close(out, ref, BF16)
    else:
        err_rel = float((out.double().cpu() - ref).abs().max() / ref.abs().max())
        assert err_rel <= 4e-7 * math.sqrt(K), err_rel
    # every tile width gives the same sums (one order of accumulation over K); the narrow
    # ones leave by plain stores, multiples of 64 columns through shared memory and TMA stores
    for bn in (32, 160, 192, 256):
        other = torch.empty_like(out)
        assert ops.gemm_bf16_pair(x, w, other, err, bn=bn)
        assert torch.equal(other, out), f"tile width {bn} changes the result"
    assert int(err.item()) == 0


@pytest.mark.parametrize("M,N,K", [(5, 96, 64), (300, 1000, 520), (1024, 4096, 2048),
                                   (700, 2050, 72)])
def test_gemm_bf16_pair_adds_into_a_float_matrix(cuda_device, M, N, K):
    """``out += x w^T``: every element gets its sum once (through TMA reductions where the rows
    start on 16-byte boundaries, by plain read-add-write otherwise), rows and columns beyond
    the matrix are not touched, and a second call adds again."""
    from binfer_b200.csrc import ops
    g = torch.Generator().manual_seed(M + N)
    x = torch.randn(M, K, generator=g).to(BF16).to(cuda_device)
    w = (0.05 * torch.randn(N, K, generator=g)).to(BF16).to(cuda_device)
    base = torch.randn(M + 3, N, generator=g).to(cuda_device)
    buf = base.clone()
    err = ops.error_word(cuda_device)
    assert ops.gemm_bf16_pair(x, w, buf[:M], err, accumulate=True)
    assert int(err.item()) == 0
    prod = x.double().cpu() @ w.double().cpu().T
    ref = base[:M].double().cpu() + prod
    got = buf[:M].double().cpu()
    assert float((got - ref).abs().max() / ref.abs().max()) <= 4e-7 * math.sqrt(K) + 1e-6
    assert torch.equal(buf[M:], base[M:])
    assert ops.gemm_bf16_pair(x, w, buf[:M], err, accumulate=True)
    ref2 = ref + prod
    assert float((buf[:M].double().cpu() - ref2).abs().max() / ref2.abs().max()) \
        <= 8e-7 * math.sqrt(K) + 1e-6
    assert int(err.item()) == 0


@pytest.mark.parametrize("M,I,K", [(3, 96, 64), (256, 12288, 1024), (300, 1000, 520),
                                   (1100, 3000, 2048), (129, 72, 4104), (2048, 1536, 4096)])
def test_gemm_bf16_pair_gated(cuda_device, M, I, K):
    """The stacked gate/up product with the activation in its epilogue: every output column
    pairs its gate row with the up row of the same output, at widths that are no multiple of
    the tile; the rows beyond a partial tile stay untouched."""
    from binfer_b200.csrc import ops
    g = torch.Generator().manual_seed(M + I)
    x = torch.randn(M, K, generator=g).to(BF16).to(cuda_device)
    w = (0.05 * torch.randn(2 * I, K, generator=g)).to(BF16).to(cuda_device)
    w[I:] *= torch.linspace(0.5, 2.0, I, device=cuda_device).to(BF16).unsqueeze(1)   # up rows differ
    buf = torch.full((M + 2, I), 99.0, device=cuda_device, dtype=BF16)
    out = buf[:M]
    err = ops.error_word(cuda_device)
    assert ops.gemm_bf16_pair(x, w, out, err, gated=True)
    assert int(err.item()) == 0
    gu = x.double().cpu() @ w.double().cpu().T
    ref = gu[:, :I] / (1 + torch.exp(-gu[:, :I])) * gu[:, I:]
    _close(out, ref, BF16)
    assert float(buf[M:].float().min()) == 99.0
    for bn in (64, 192, 256):
        other = torch.empty_like(out)
        assert ops.gemm_bf16_pair(x, w, other, err, bn=bn, gated=True)
        assert torch.equal(other, out), f"tile width {bn} changes the result"
    assert int(err.item()) == 0


def test_gemm_bf16_refuses_what_it_cannot_take(cuda_device):
    from binfer_b200.csrc import ops
    x = torch.randn(4, 100, device=cuda_device).to(BF16)       # K not a multiple of 8
    w = torch.randn(32, 100, device=cuda_device).to(BF16)
    out = torch.full((4, 32), 5.0, device=cuda_device, dtype=BF16)
    assert not ops.gemm_bf16(x, w, out, ops.error_word(cuda_device))
    assert bool((out == 5.0).all())


def test_engine_with_own_gemm_everywhere(cuda_device, tmp_path):
    """The bfloat16 engine with every product on the tcgen05 kernel still matches the plain
    implementation (config with hidden sizes that are multiples of 8)."""
    import helpers as H
    from binfer_b200.engine import make_env, make_runner, model_from_dir
    import importlib
    L = importlib.import_module("binfer_b200.parts.linear")
    d = H.make_model_dir(tmp_path, "B", BF16)
    raw, w = H.read_model_dir(d)
    reqs = {f"r{i}": H.random_tokens(n, raw["vocab_size"], n) for i, n in enumerate([70, 150, 9])}
    ref = {rid: P.forward(raw, w, t, torch.float64) for rid, t in reqs.items()}
    before = L._POLICY
    L.set_gemm_policy("own")
    try:
        env = make_env(BF16)
        steps = H.trace_mixed(reqs)
        runner = make_runner(model_from_dir(d, env), env, page_size=8,
                             num_pages=H.peak_pages(steps, 8))
        got = H.run_trace(runner, steps)
    finally:
        L.set_gemm_policy(before)
    worst = max(H.rel_err(row, ref[rid][p]) for (rid, p), row in got.items())
    assert worst <= 3e-2, worst


@pytest.mark.parametrize("nh,nkv,d,ps,window,spike", [
    (4, 2, 32, 16, None, False), (6, 1, 32, 8, None, True), (8, 2, 128, 16, None, True),
    (5, 5, 96, 4, 24, True), (3, 3, 64, 5, 70, True), (2, 1, 256, 16, 100, True),
    (4, 4, 128, 64, 130, True), (6, 2, 128, 8, None, True), (4, 1, 64, 32, 150, True)])
@pytest.mark.parametrize("variant", ["mma_sync", "umma", "umma2"])
def test_prefill_attention_over_pages(cuda_device, nh, nkv, d, ps, window, spike, variant):
    """Portions that start in the middle of a prompt, straddle 64-key tiles and pages, next to
    whole prompts; the far key and the window's edge are made to stand out."""
    from binfer_b200.csrc import ops
    if variant == "umma" and not (d in (64, 128) and ps >= 8 and 64 % ps == 0):
        pytest.skip("the umma variant does not take this head or page size")
    if variant == "umma2" and not (d == 128 and ps >= 8 and 64 % ps == 0):
        pytest.skip("the umma2 variant does not take this head or page size")
    ctxs, qlens = [70, 200, 129, 300, 64, 2, 400], [70, 37, 5, 130, 64, 2, 290]
    q, kc, vc, sot, pos, bt, ref = _attention_case(cuda_device, BF16, nh, nkv, d, ps, ctxs,
                                                   qlens, window, spike, seed=11)
    items, row = [], 0
    for b, (n, ql) in enumerate(zip(ctxs, qlens)):
        items.append([b, row, ql, n - ql])
        row += ql
    items = torch.tensor(items, dtype=torch.int32, device=cuda_device)
    out = torch.zeros_like(q)
    err = _err(cuda_device)
    ops.prefill_attention(q, kc, vc, items, len(ctxs), max(qlens), bt, out, nh, nkv, d, window,
                          d ** -0.5, err, variant=variant)
    assert int(err.item()) == 0
    _close(out, ref, BF16)
    # a subset of the portions leaves the other rows alone
    out2 = torch.zeros_like(q)
    ops.prefill_attention(q, kc, vc, items[1:3].contiguous(), 2, 37, bt, out2, nh, nkv, d,
                          window, d ** -0.5, err, variant=variant)
    assert torch.equal(out2[70:112], out[70:112]) and float(out2[:70].abs().max()) == 0.0


@pytest.mark.parametrize("nh,nkv,ps,cap,splits", [(4, 2, 16, 3.0, 1), (6, 6, 8, 0.7, 3),
                                                   (2, 1, 64, 0.0, 1), (8, 2, 16, 5.0, 2)])
def test_prefill_attention_soft_cap_into_a_column_block(cuda_device, nh, nkv, ps, cap, splits):
    """The umma2 variant with scores through ``c tanh(s / c)``, the result times a factor and
    written into a column block of a wider buffer whose other columns stay as they were, with
    and without the keys shared out.  The scores are large, so a cap left out would show."""
    from binfer_b200.csrc import ops
    dev, d, gen = cuda_device, 128, torch.Generator().manual_seed(nh * 10 + ps)
    ctxs, qlens = [300, 70, 1100, 2, 257], [300, 37, 260, 2, 129]
    scale, factor, left, right = 0.5, 0.8, 16, 8
    kcs, vcs, tables, qs, refs, items, base, row = [], [], [], [], [], [], 0, 0
    for b, (n, ql) in enumerate(zip(ctxs, qlens)):
        k = torch.randn(n, nkv, d, generator=gen).to(BF16).double()
        v = torch.randn(n, nkv, d, generator=gen).to(BF16).double()
        q = torch.randn(ql, nh, d, generator=gen).to(BF16).double()
        kh = k.repeat_interleave(nh // nkv, dim=1)
        vh = v.repeat_interleave(nh // nkv, dim=1)
        sc = torch.einsum("qhd,nhd->hqn", q, kh) * scale
        if cap > 0:
            sc = cap * torch.tanh(sc / cap)
        seen = torch.arange(n)[None, :] <= (n - ql + torch.arange(ql))[:, None]
        sc = sc.masked_fill(~seen[None], float("-inf"))
        refs.append(factor * torch.einsum("hqn,nhd->qhd", torch.softmax(sc, dim=-1), vh))
        kc, vc, ids = _paged(k, v, ps, "cpu", BF16, 70 + b, False)
        kcs.append(kc)
        vcs.append(vc)
        tables.append([i + base for i in ids])
        base += kc.shape[0]
        qs.append(q)
        items.append([b, row, ql, n - ql])
        row += ql
    bt = torch.zeros(len(ctxs), max(len(t) for t in tables), dtype=torch.int32)
    for b, t in enumerate(tables):
        bt[b, :len(t)] = torch.tensor(t, dtype=torch.int32)
    q_all = torch.cat(qs).to(BF16).reshape(row, nh * d).to(dev)
    items = torch.tensor(items, dtype=torch.int32, device=dev)
    wide = torch.full((row, left + nh * d + right), 7.0, dtype=BF16, device=dev)
    out = wide[:, left:left + nh * d]
    kc, vc = torch.cat(kcs).to(dev), torch.cat(vcs).to(dev)
    assert ops.prefill_attention_takes_capped(q_all, kc, d, d)
    err = _err(dev)
    ops.prefill_attention(q_all, kc, vc, items, len(ctxs), max(qlens), bt.to(dev), out, nh, nkv,
                          d, None, scale, err, variant="umma2", splits=splits, softcap=cap,
                          out_scale=factor)
    assert int(err.item()) == 0
    _close(out, torch.cat(refs).reshape(row, nh * d), BF16)
    assert bool((wide[:, :left] == 7.0).all()) and bool((wide[:, left + nh * d:] == 7.0).all())
    if cap > 0:
        plain = torch.empty((row, nh * d), dtype=BF16, device=dev)
        ops.prefill_attention(q_all, kc, vc, items, len(ctxs), max(qlens), bt.to(dev), plain, nh,
                              nkv, d, None, scale, err, variant="umma2", splits=splits)
        assert float((plain.float() * factor - out.float()).abs().max()) > 0.05


@pytest.mark.parametrize("splits", [2, 3, 8])
@pytest.mark.parametrize("ps,neighbours", [(16, True), (8, False), (64, False)])
def test_prefill_attention_keys_shared_out(cuda_device, splits, ps, neighbours):
    """Few queries after many cached keys: the keys of a block of 256 queries are shared out
    over several CTAs and merged.  Portions whose blocks have fewer key tiles than there are
    shares (an empty share), rows that see no key of a share (causal), a portion of two rows,
    and one from position 0, beside long prefixes; the far key is made to stand out."""
    from binfer_b200.csrc import ops
    nh, nkv, d = 4, 2, 128
    ctxs, qlens = [1500, 70, 2100, 2, 900], [200, 70, 300, 2, 129]
    q, kc, vc, sot, pos, bt, ref = _attention_case(cuda_device, BF16, nh, nkv, d, ps, ctxs,
                                                   qlens, None, True, seed=31,
                                                   neighbours=neighbours)
    items, row = [], 0
    for b, (n, ql) in enumerate(zip(ctxs, qlens)):
        items.append([b, row, ql, n - ql])
        row += ql
    items = torch.tensor(items, dtype=torch.int32, device=cuda_device)
    err = _err(cuda_device)
    out = torch.zeros_like(q)
    ops.prefill_attention(q, kc, vc, items, len(ctxs), max(qlens), bt, out, nh, nkv, d, None,
                          d ** -0.5, err, variant="umma2", splits=splits)
    assert int(err.item()) == 0
    _close(out, ref, BF16)
    # the number of shares chosen from the longest context gives the same values to rounding
    auto = torch.zeros_like(q)
    ops.prefill_attention(q, kc, vc, items, len(ctxs), max(qlens), bt, auto, nh, nkv, d, None,
                          d ** -0.5, err, max_ctx=max(ctxs))
    assert int(err.item()) == 0
    _close(auto, ref, BF16)


@pytest.mark.parametrize("seed", [1, 2, 3, 4, 5, 6])
def test_prefill_attention_random_shapes(cuda_device, seed):
    """Shapes drawn at random (heads, groups, page size, window, how many portions, where they
    start and how long they are, pages side by side or scattered): the kernel that the policy
    picks, with the keys shared out or not as it decides, against the plain result."""
    import random
    from binfer_b200.csrc import ops
    rnd = random.Random(seed)
    nkv = rnd.choice([1, 2, 4])
    nh = nkv * rnd.choice([1, 2, 4, 7])
    d, ps = 128, rnd.choice([8, 16, 32, 64])
    window = rnd.choice([None, None, rnd.randint(40, 900)])
    n = rnd.randint(1, 4)
    qlens = [rnd.choice([2, rnd.randint(3, 130), rnd.randint(131, 700)]) for _ in range(n)]
    ctxs = [ql + rnd.choice([0, rnd.randint(1, 300), rnd.randint(1500, 3000)]) for ql in qlens]
    q, kc, vc, sot, pos, bt, ref = _attention_case(cuda_device, BF16, nh, nkv, d, ps, ctxs,
                                                   qlens, window, True, seed=100 + seed,
                                                   neighbours=rnd.random() < 0.5)
    items, row = [], 0
    for b, (c, ql) in enumerate(zip(ctxs, qlens)):
        items.append([b, row, ql, c - ql])
        row += ql
    items = torch.tensor(items, dtype=torch.int32, device=cuda_device)
    err = _err(cuda_device)
    out = torch.zeros_like(q)
    ops.prefill_attention(q, kc, vc, items, n, max(qlens), bt, out, nh, nkv, d, window,
                          d ** -0.5, err, max_ctx=max(ctxs))
    assert int(err.item()) == 0
    _close(out, ref, BF16)
    two = torch.zeros_like(q)
    ops.prefill_attention(q, kc, vc, items, n, max(qlens), bt, two, nh, nkv, d, window,
                          d ** -0.5, err, variant="umma2", splits=1)
    assert int(err.item()) == 0
    _close(two, ref, BF16)


@pytest.mark.parametrize("ps,window,neighbours", [(64, None, False), (16, 300, False),
                                                  (8, None, False), (16, None, True),
                                                  (8, 300, True), (32, 100, True)])
@pytest.mark.parametrize("variant", ["umma", "umma2"])
def test_prefill_attention_long_portions(cuda_device, ps, window, neighbours, variant):
    """Portions of many query tiles over many key tiles (the rings of stages wrap, the two
    query tiles of a block end on different key tiles), from the start of a prompt and from
    its middle, with and without a window; over shuffled pages and over pages that lie side
    by side in the pool, whose tiles come as one box (but for the tile a window cuts)."""
    from binfer_b200.csrc import ops
    nh, nkv, d = 4, 2, 128
    ctxs, qlens = [1500, 700, 1100], [900, 700, 257]
    q, kc, vc, sot, pos, bt, ref = _attention_case(cuda_device, BF16, nh, nkv, d, ps, ctxs,
                                                   qlens, window, True, seed=23,
                                                   neighbours=neighbours)
    items, row = [], 0
    for b, (n, ql) in enumerate(zip(ctxs, qlens)):
        items.append([b, row, ql, n - ql])
        row += ql
    items = torch.tensor(items, dtype=torch.int32, device=cuda_device)
    out = torch.zeros_like(q)
    err = _err(cuda_device)
    ops.prefill_attention(q, kc, vc, items, len(ctxs), max(qlens), bt, out, nh, nkv, d, window,
                          d ** -0.5, err, variant=variant)
    assert int(err.item()) == 0
    _close(out, ref, BF16)


@pytest.mark.parametrize("far", [40, 70, 130, 200, 390])
@pytest.mark.parametrize("variant", ["mma_sync", "umma", "umma2"])
def test_prefill_attention_when_one_key_dwarfs_the_tiles_before_it(cuda_device, variant, far):
    """A score hundreds above everything in earlier key tiles: what those tiles have left in the
    output counts nothing any more (the factor on it underflows to zero)."""
    from binfer_b200.csrc import ops
    nh, nkv, d, ps, n = 4, 2, 128, 16, 400
    g = torch.Generator().manual_seed(far)
    q, k, v = (torch.randn(n, h, d, generator=g).to(BF16).double() for h in (nh, nkv, nkv))
    k[far] = 0
    k[far, :, 0] = 128.0
    q[-1, :, 0] = 64.0                      # a score of 724
    kc, vc, ids = _paged(k, v, ps, "cpu", BF16, 3)
    ref = P.causal_attention(q, k, v, d ** -0.5, None).reshape(n, nh * d)
    qd = q.to(BF16).reshape(n, nh * d).to(cuda_device)
    bt = torch.tensor([ids], dtype=torch.int32, device=cuda_device)
    items = torch.tensor([[0, 0, n, 0]], dtype=torch.int32, device=cuda_device)
    out = torch.zeros_like(qd)
    err = _err(cuda_device)
    ops.prefill_attention(qd, kc.to(cuda_device), vc.to(cuda_device), items, 1, n, bt, out, nh,
                          nkv, d, None, d ** -0.5, err, variant=variant)
    assert int(err.item()) == 0
    _close(out[-1:], ref[-1:], BF16)
    _close(out, ref, BF16)


@pytest.mark.parametrize("M,N,K,bn,c", [(1, 300, 520, 64, 4), (8, 4096, 4096, 128, 4),
                                        (16, 1000, 4104, 128, 8), (7, 6144, 4096, 192, 4),
                                        (3, 256, 256, 256, 2), (16, 4096, 12288, 128, 4),
                                        (5, 96, 64, 64, 4), (8, 24576, 4096, 176, 1),
                                        (2, 1000, 320, 80, 1), (17, 4096, 4096, 128, 4),
                                        (40, 520, 1024, 64, 2), (64, 4096, 12288, 128, 4),
                                        (33, 6144, 4096, 192, 4)])
@pytest.mark.parametrize("out_dtype", [BF16, F32])
def test_gemm_bf16_cluster_split_k(cuda_device, M, N, K, bn, c, out_dtype):
    """K split over a cluster and reduced through distributed shared memory; widths and depths
    that are no multiple of the tile, fewer K steps than CTAs in the cluster."""
    from binfer_b200.csrc import ops
    g = torch.Generator().manual_seed(M * 3 + N)
    x = torch.randn(M, K, generator=g).to(BF16).to(cuda_device)
    w = (0.05 * torch.randn(N, K, generator=g)).to(BF16).to(cuda_device)
    out = torch.full((M, N), 99.0, device=cuda_device, dtype=out_dtype)
    err = ops.error_word(cuda_device)
    assert ops.gemm_bf16_cluster(x, w, out, err, bn, c)
    assert int(err.item()) == 0
    ref = x.double().cpu() @ w.double().cpu().T
    if out_dtype == BF16:
        _close(out, ref, BF16)
    else:
        err_rel = float((out.double().cpu() - ref).abs().max() / ref.abs().max())
        assert err_rel <= 4e-7 * math.sqrt(K), err_rel
    again = torch.empty_like(out)
    assert ops.gemm_bf16_cluster(x, w, again, err, bn, c)
    assert torch.equal(again, out), "the split-K sum must have one fixed order"
    assert not ops.gemm_bf16_cluster(torch.zeros(65, K, device=cuda_device, dtype=BF16), w,
                                     torch.empty(65, N, device=cuda_device, dtype=out_dtype),
                                     err, bn, c)


@pytest.mark.parametrize("N,K,bn,c", [(5120, 25600, 192, 4), (5120, 8192, 192, 4)])
def test_gemm_bf16_cluster_many_k_steps_many_launches(cuda_device, N, K, bn, c):
    """A hundred K steps per CTA through a ring of seven slots, two issuing threads, a
    thousand launches: every launch gives the first one's bits and no wait gives up.  (Each
    ring slot has one issuer: were the K steps dealt out in turn, a thread would wait for
    every second fill of a slot with the same parity, which held only while the copies
    landed in order.  The Qwen3-32B shape's output and down projections are these sizes.)"""
    from binfer_b200.csrc import ops
    g = torch.Generator().manual_seed(N + K)
    x = torch.randn(8, K, generator=g).to(BF16).to(cuda_device)
    w = (0.05 * torch.randn(N, K, generator=g)).to(BF16).to(cuda_device)
    err = ops.error_word(cuda_device)
    first = torch.empty((8, N), device=cuda_device, dtype=BF16)
    assert ops.gemm_bf16_cluster(x, w, first, err, bn, c)
    _close(first, x.double().cpu() @ w.double().cpu().T, BF16)
    out = torch.empty_like(first)
    same = torch.ones((), dtype=torch.bool, device=cuda_device)
    for _ in range(1000):
        assert ops.gemm_bf16_cluster(x, w, out, err, bn, c)
        same &= (out == first).all()
    assert bool(same) and int(err.item()) == 0


# ------------------------------------------------------------ recurrences in chunks of tokens
def _walk64(q, k, v, decay, S):
    """``S <- decay S + k v^T, o = S^T q`` in float64: (o, S)."""
    out = torch.empty_like(v)
    for t in range(v.shape[0]):
        S = S * decay[t][:, None, None] + k[t][:, :, None] * v[t][:, None, :]
        out[t] = (q[t][:, None, :] @ S)[:, 0]
    return out, S


# portions at the edges of a chunk of 64 and of the shortest portion that has chunks, beside
# portions that are walked; sizes below, at and between tiles of 64; shared q and k; a fixed decay;
# decays that are zero
@pytest.mark.parametrize("lens,H,G,dk,dv,decays", [
    ([161, 1, 192, 160, 257], 4, 2, 32, 24, "spread"), ([193, 320], 3, 3, 20, 68, "zeros"),
    ([300], 2, 1, 128, 64, "slow"), ([170, 3], 2, 2, 68, 132, "fixed")])
def test_linear_scan_in_chunks(cuda_device, lens, H, G, dk, dv, decays):
    from binfer_b200.csrc import ops
    torch.manual_seed(len(lens) + dk)
    T, B, dev = sum(lens), len(lens), cuda_device
    qk = torch.randn(T, 2, G, dk, device=dev)
    v = torch.randn(T, H, dv, device=dev)
    d = torch.rand(T, H, device=dev)
    if decays == "slow":
        d = 1.0 - 0.01 * d
    elif decays == "zeros":
        d[torch.rand(T, H, device=dev) < 0.1] = 0.0
    elif decays == "fixed":
        d = d[:1].expand(T, H).contiguous()
    state = torch.randn(B + 1, H * dk * dv, device=dev)
    slots = torch.arange(B, dtype=torch.int32, device=dev).flip(0).contiguous()
    qs = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=dev)
    out = torch.full((T, H * dv), 7.0, device=dev)
    got, err = state.clone(), _err(dev)
    ops.linear_scan(qk, v, d, got, qs, slots, out, B, H, G, dk, dv, err, max_q=max(lens),
                    chunked=True)
    assert int(err.item()) == 0 and torch.equal(got[B], state[B])
    for b in range(B):
        a, e, s = int(qs[b]), int(qs[b + 1]), int(slots[b])
        q, k = (qk[a:e, i].double().repeat_interleave(H // G, 1) for i in (0, 1))
        S0 = state[s].double().view(H, dv, dk).transpose(1, 2)
        o, S = _walk64(q, k, v[a:e].double(), d[a:e].double(), S0)
        # the same recurrence over absolute values bounds what a relative error of every factor and
        # sum can come to: sums of runs of 16 and of up to 12 + 4 runs, a weight (two roundings),
        # one update per chunk
        bound_o, bound_S = _walk64(q.abs(), k.abs(), v[a:e].double().abs(), d[a:e].double(), S0.abs())
        c = (64 + 4 * len(lens)) * 2.0 ** -24
        assert bool(((out[a:e].view(-1, H, dv).double() - o).abs() <= c * bound_o + 1e-30).all())
        have = got[s].double().view(H, dv, dk).transpose(1, 2)
        assert bool(((have - S).abs() <= c * bound_S + 1e-30).all())
    # a bad slot is flagged, and every state that no request owns left alone
    bad, keep = slots.clone(), got.clone()
    bad[0] = B + 5
    ops.linear_scan(qk, v, d, keep, qs, bad, out, B, H, G, dk, dv, err, max_q=max(lens),
                    chunked=True)
    assert int(err.item()) == 2 and torch.equal(keep[int(slots[0])], got[int(slots[0])])
    err.zero_()


# the same on the tensor cores: two heads of 64 a tile and one of 128 or more, requests of odd lengths beside
# walked ones, more tiles than SMs; the multiply-adds beside them
@pytest.mark.parametrize("lens,H,G,dk,dv,decays", [
    ([161, 1, 192, 160, 257], 4, 2, 128, 64, "spread"), ([193, 320], 4, 1, 256, 64, "zeros"),
    ([300], 2, 2, 128, 128, "slow"), ([170, 3, 700], 16, 8, 128, 256, "slow")])
def test_linear_chunks_on_tensor_cores(cuda_device, monkeypatch, lens, H, G, dk, dv, decays):
    """Bound as in test_linear_scan_in_chunks; and no further from float64 than the multiply-adds with slow
    decays, half a unit in the last place more with others (a sum of few terms is cut where that one rounds)."""
    from binfer_b200.csrc import ops
    torch.manual_seed(len(lens) + dk)
    T, B, dev = sum(lens), len(lens), cuda_device
    qk, v = torch.randn(T, 2, G, dk, device=dev), torch.randn(T, H, dv, device=dev)
    d = torch.rand(T, H, device=dev)
    if decays == "slow":
        d = 1.0 - 0.01 * d
    elif decays == "zeros":
        d[torch.rand(T, H, device=dev) < 0.1] = 0.0
    state = torch.randn(B + 1, H * dk * dv, device=dev)
    slots = torch.arange(B, dtype=torch.int32, device=dev).flip(0).contiguous()
    qs = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=dev)
    got, err = [], _err(dev)
    for ctas in (0, 1 << 30):
        monkeypatch.setattr(ops, "LINEAR_TENSOR_MIN_CTAS", ctas)
        _, terms = ops._chunk_scratch(True, max(lens), T, B, H, G, dk, dv, state, 0, qk)
        assert terms == (ctas == 0)
        s, o = state.clone(), torch.full((T, H * dv), 7.0, device=dev)
        ops.linear_scan(qk, v, d, s, qs, slots, o, B, H, G, dk, dv, err, max_q=max(lens), chunked=True)
        assert int(err.item()) == 0 and torch.equal(s[B], state[B])
        got.append((o, s))
    off = [[0.0, 0.0], [0.0, 0.0]]
    for b in range(B):
        a, e, at = int(qs[b]), int(qs[b + 1]), int(slots[b])
        q, k = (qk[a:e, i].double().repeat_interleave(H // G, 1) for i in (0, 1))
        S0 = state[at].double().view(H, dv, dk).transpose(1, 2)
        o, S = _walk64(q, k, v[a:e].double(), d[a:e].double(), S0)
        bound_o, bound_S = _walk64(q.abs(), k.abs(), v[a:e].double().abs(), d[a:e].double(), S0.abs())
        c = (64 + 4 * len(lens)) * 2.0 ** -24
        for i, (go, gs) in enumerate(got):
            oo = go[a:e].view(-1, H, dv).double()
            SS = gs[at].double().view(H, dv, dk).transpose(1, 2)
            assert bool(((oo - o).abs() <= c * bound_o + 1e-30).all())
            assert bool(((SS - S).abs() <= c * bound_S + 1e-30).all())
            if e - a > ops.CHUNK_SCAN_MIN:
                for j, (x, y) in enumerate(((oo, o), (SS, S))):
                    off[i][j] = max(off[i][j], float((x - y).norm() / y.norm()))
    for tensor, adds in zip(*off):
        assert tensor <= adds + (0.0 if decays == "slow" else 2.0 ** -25), off
    bad, keep, o = slots.clone(), got[0][1].clone(), got[0][0].clone()
    bad[0] = B + 5
    monkeypatch.setattr(ops, "LINEAR_TENSOR_MIN_CTAS", 0)
    ops.linear_scan(qk, v, d, keep, qs, bad, o, B, H, G, dk, dv, err, max_q=max(lens), chunked=True)
    assert int(err.item()) == 2 and torch.equal(keep[int(slots[0])], got[0][1][int(slots[0])])
    err.zero_()


# (the delta rule's own sums leave float's range before these do)
@pytest.mark.parametrize("kind,dv,what", [
    (*k, w) for k in (("linear", 64), ("linear", 128), ("delta", 128))
    for w in ("v", "k", "q", "decay", "state", "large v", "small", "products", "all v")
    if k[0] == "linear" or w not in ("large v", "products", "state")])
def test_chunks_on_tensor_cores_take_floats_of_every_size(cuda_device, monkeypatch, kind, dv, what):
    """Infinities, NaN, floats that have no terms, products that leave float's range: numbers where the
    multiply-adds have numbers, the same ones but for rounding; the bits of the tokens before are the clean
    call's."""
    from binfer_b200.csrc import ops
    monkeypatch.setattr(ops, "DELTA_CHUNK_MIN", 160)
    dev, T, H, G, dk, at = cuda_device, 330, 4, 2, 128, 140
    torch.manual_seed(11)
    unit = lambda x: torch.nn.functional.normalize(x, dim=-1)
    qs = torch.tensor([0, T], dtype=torch.int32, device=dev)
    slots, err, outs = torch.zeros(1, dtype=torch.int32, device=dev), _err(dev), {}
    clean = (unit(torch.randn(T, 2, G, dk, device=dev)), torch.randn(T, H, dv, device=dev),
             1 - 0.1 * torch.rand(T, H, device=dev), 0.1 * torch.randn(1, H * dk * dv, device=dev))
    for bad in (False, True):
        x, v, d, s0 = (t.clone() for t in clean)
        if bad and what == "v":
            v[at, 1, 5] = float("inf")
        elif bad and what == "all v":
            v[:] = float("inf")
        elif bad and what == "k":
            x[at, 1, 0, 77] = float("-inf")
        elif bad and what == "q":
            x[at, 0, 1, 3] = float("nan")
        elif bad and what == "decay":
            d[at, 2] = float("nan")
        elif bad and what == "state":
            s0[0, 5000] = float("inf")
        elif bad and what == "large v":
            v[at:, 1] *= 3e37
        elif bad and what == "small":
            v *= 1e-33
            s0 *= 1e-33
        elif bad and what == "products":
            v[at:, 1], x[at:, 1, 0] = v[at:, 1] * 1e24, x[at:, 1, 0] * 1e24
        for ctas in (0, 1 << 30):
            monkeypatch.setattr(ops, "LINEAR_TENSOR_MIN_CTAS", ctas)
            monkeypatch.setattr(ops, "CHUNK_SCAN_MAX_BYTES", 768 << 20)
            if kind == "delta" and ctas:         # (the limit between the two calls' scratch)
                fn = ops.lib().bf_chunk_scan_delta_scratch
                args = [ops._c_int(z) for z in (T, 1, H, G, dk, dv, 0, 0)]
                monkeypatch.setattr(ops, "CHUNK_SCAN_MAX_BYTES", fn(*args))
            assert (_delta_on_tensor_cores(T, 1, H, G, dk, dv) if kind == "delta" else
                    ops._chunk_scratch(True, T, T, 1, H, G, dk, dv, s0, 0)[1]) == (ctas == 0)
            s, o = s0.clone(), torch.empty(T, H * dv, device=dev)
            if kind == "linear":
                ops.linear_scan(x, v, d, s, qs, slots, o, 1, H, G, dk, dv, err, max_q=T, chunked=True)
            else:
                qkv = torch.cat([x[:, 0].reshape(T, -1), x[:, 1].reshape(T, -1), v.reshape(T, -1)], 1).contiguous()
                ops.delta_scan(qkv, torch.stack([d / 2, d], 1).contiguous(), s, qs, slots, o, 1, H, G, dk, dv, err,
                               max_q=T, chunked=True)
            outs[bad, ctas == 0] = (o.view(T, H, dv), s)
    assert int(err.item()) == 0
    for mine, adds in zip(outs[True, True], outs[True, False]):
        assert torch.equal(mine.isfinite(), adds.isfinite())
        fin = mine.isfinite()
        if bool(fin.any()):
            scale = adds[fin].abs().max()
            assert float(((mine - adds)[fin] / scale).abs().max()) <= 1e-5
    if what not in ("state", "small", "all v"):
        assert torch.equal(outs[True, True][0][:at], outs[False, True][0][:at])


@pytest.mark.parametrize("dv", [64, 128])
def test_numbers_without_terms_four_chunks_apart(cuda_device, monkeypatch, dv):
    """One value size has a float without terms in every fourth chunk, and a decay of zero forgets it: the flags of
    those chunks share a place.  Between the zeros the results are the multiply-adds' but for rounding (chains of at
    most 700 + 128 sums, twice: 2^-24 each, a tenth of that where they err at random)."""
    from binfer_b200.csrc import ops
    dev, T, H, G, dk = cuda_device, 700, 4, 2, 128
    torch.manual_seed(13)
    qk = torch.nn.functional.normalize(torch.randn(T, 2, G, dk, device=dev), dim=-1)
    v, d = torch.randn(T, H, dv, device=dev), 1 - 0.1 * torch.rand(T, H, device=dev)
    for at in (70, 326, 582):                    # in chunks 1, 5 and 9
        v[at, 1, 5], d[at + 40, 1] = 3e31, 0.0
    qs, slots = torch.tensor([0, T], dtype=torch.int32, device=dev), torch.zeros(1, dtype=torch.int32, device=dev)
    got, err = [], _err(dev)
    for ctas in (0, 1 << 30):
        monkeypatch.setattr(ops, "LINEAR_TENSOR_MIN_CTAS", ctas)
        s, o = torch.zeros(1, H * dk * dv, device=dev), torch.empty(T, H * dv, device=dev)
        assert ops._chunk_scratch(True, T, T, 1, H, G, dk, dv, s, 0, qk)[1] == (ctas == 0)
        ops.linear_scan(qk, v, d, s, qs, slots, o, 1, H, G, dk, dv, err, max_q=T, chunked=True)
        got.append((o.view(T, H, dv), s))
    assert int(err.item()) == 0
    for a, e in ((0, 70), (70, 110), (110, 326), (326, 366), (366, 582), (582, 622), (622, T)):
        x, y = (o[a:e] for o, _ in got)
        for part in ((slice(None), 1, 5), (slice(None), 0), (slice(None), 1, slice(6, None))):
            assert bool(y[part].isfinite().all()) and float(y[part].norm()) > 0
            assert float((x[part] - y[part]).norm() / y[part].norm()) <= 1e-5, (a, part)
    assert float((got[0][1] - got[1][1]).norm() / got[1][1].norm()) <= 1e-5


def test_linear_chunks_on_tensor_cores_of_many_tiles(cuda_device, monkeypatch):
    """More tiles than one CTA an SM has room for in its list: the multiply-adds' results."""
    from binfer_b200.csrc import ops
    dev, T, H, dk, dv = cuda_device, 9700, 64, 128, 128
    torch.manual_seed(12)
    qk = torch.nn.functional.normalize(torch.randn(T, 2, 8, dk, device=dev), dim=-1)
    v, d = torch.randn(T, H, dv, device=dev), 1 - 0.05 * torch.rand(T, H, device=dev)
    qs, slots = torch.tensor([0, T], dtype=torch.int32, device=dev), torch.zeros(1, dtype=torch.int32, device=dev)
    got, err = [], _err(dev)
    monkeypatch.setattr(ops, "CHUNK_SCAN_MAX_BYTES", 2 << 30)
    for ctas in (0, 1 << 30):
        monkeypatch.setattr(ops, "LINEAR_TENSOR_MIN_CTAS", ctas)
        s, o = torch.zeros(1, H * dk * dv, device=dev), torch.empty(T, H * dv, device=dev)
        assert ops._chunk_scratch(True, T, T, 1, H, 8, dk, dv, s, 0)[1] == (ctas == 0)
        ops.linear_scan(qk, v, d, s, qs, slots, o, 1, H, 8, dk, dv, err, max_q=T, chunked=True)
        got.append((o, s))
    assert int(err.item()) == 0
    for a, b in zip(*got):
        assert float((a - b).norm() / b.norm()) <= 5e-7


def test_retention_part_walks_decays_below_zero(cuda_device, monkeypatch):
    """A portion long enough for chunks and the same tokens in two that are walked."""
    from types import SimpleNamespace
    from binfer_b200.config import RetentionSpec
    from binfer_b200.csrc import ops
    from binfer_b200.engine import make_env
    from binfer_b200.parts.retention import RetentionMixer
    monkeypatch.setattr(ops, "chunk_scan_pays", lambda *a: True)
    dev, T = cuda_device, 2 * ops.CHUNK_SCAN_MIN
    spec = RetentionSpec(num_heads=2, qk_dim=16, v_dim=128, decays=(-0.9, 0.8), position=None,
                         norm_eps=1e-5)
    mixer = RetentionMixer(spec, 64, "", make_env(BF16))
    torch.manual_seed(3)
    proj = torch.randn(T, mixer.in_rows, device=dev).to(BF16)
    got = []
    for cuts in ([T], [T // 2, T // 2]):
        view = SimpleNamespace(state=torch.zeros(1, 2 * 16 * 128, device=dev))
        ys = []
        for x in proj.split(cuts):
            n, out = x.shape[0], torch.empty(x.shape[0], mixer.out_cols, dtype=BF16, device=dev)
            ctx = SimpleNamespace(positions=torch.arange(n, dtype=torch.int32, device=dev),
                                  q_start=torch.tensor([0, n], dtype=torch.int32, device=dev),
                                  state_slots=torch.zeros(1, dtype=torch.int32, device=dev), B=1,
                                  decode_only=False, max_q_len=n, err=_err(dev))
            mixer.run(x, ctx, view, out, 1.0)
            ys.append(out)
        got.append((torch.cat(ys), view.state))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert bool(got[0][0].isfinite().all())


def test_chunks_pass_nan_decays_on(cuda_device):
    """A decay that is NaN shows from its token on, in the products over chunks as in the walk."""
    from binfer_b200.csrc import ops
    dev, T, H, d, at = cuda_device, 300, 2, 32, 140
    torch.manual_seed(4)
    qs = torch.tensor([0, T], dtype=torch.int32, device=dev)
    slots, err = torch.zeros(1, dtype=torch.int32, device=dev), _err(dev)
    x = torch.nn.functional.normalize(torch.randn(T, 2, H, d, device=dev), dim=-1)
    v, decay = torch.randn(T, H, d, device=dev), torch.rand(T, H, device=dev)
    decay[at, 1] = float("nan")
    for chunked in (False, True):
        out = torch.zeros(T, H * d, device=dev)
        ops.linear_scan(x, v, decay, torch.zeros(1, H * d * d, device=dev), qs, slots, out, 1, H, H,
                        d, d, err, max_q=T, chunked=chunked)
        out = out.view(T, H, d)
        assert bool(out[:, 0].isfinite().all()) and bool(out[:at, 1].isfinite().all())
        assert bool(out[at:, 1].isnan().all())


@pytest.mark.parametrize("kind", ["linear", "mlstm", "delta"])
@pytest.mark.parametrize("at", [64, 140, 255])
def test_chunks_leave_earlier_tokens_alone(cuda_device, monkeypatch, kind, at):
    """An infinite value shows from its token on: the bits of the tokens before it stay."""
    from binfer_b200.csrc import ops
    monkeypatch.setattr(ops, "DELTA_CHUNK_MIN", 160)
    dev, T, H, d = cuda_device, 300, 2, 32
    torch.manual_seed(5)
    qs = torch.tensor([0, T], dtype=torch.int32, device=dev)
    slots, err, outs = torch.zeros(1, dtype=torch.int32, device=dev), _err(dev), []
    x = torch.nn.functional.normalize(torch.randn(T, 2, H, d, device=dev), dim=-1)
    v, decay = torch.randn(T, H, d, device=dev), torch.rand(T, H, device=dev)
    for bad in (False, True):
        if bad:
            v[at, 1] = float("inf")
        out = torch.zeros(T, H * d, device=dev)
        if kind == "linear":
            ops.linear_scan(x, v, decay, torch.zeros(1, H * d * d, device=dev), qs, slots, out, 1,
                            H, H, d, d, err, max_q=T, chunked=True)
        elif kind == "delta":
            qkv = torch.cat([x.reshape(T, -1), v.reshape(T, -1)], 1).contiguous()
            gates = torch.stack([1 - decay, decay], 1).contiguous()
            ops.delta_scan(qkv, gates, torch.zeros(1, H * d * d, device=dev), qs, slots, out, 1, H,
                           H, d, d, err, max_q=T, chunked=True)
        else:
            proj = torch.cat([x.reshape(T, -1), v.reshape(T, -1)], 1).to(BF16)
            gates = torch.cat([decay, decay.log()], 1).contiguous()
            ops.mlstm_scan(proj, gates, torch.zeros(1, H, ops.mlstm_state_size(d, d), device=dev),
                           qs, slots, out, 1, H, d, d, 1.0, err, max_q=T, chunked=True)
        outs.append(out.view(T, H, d))
    clean, dirty = outs
    assert torch.equal(dirty[:, 0], clean[:, 0]) and torch.equal(dirty[:at, 1], clean[:at, 1])
    assert not bool(dirty[at, 1].isfinite().any())


def test_mlstm_chunks_take_shut_gates(cuda_device):
    """A log forget gate of -inf forgets what came before, a log input gate of -inf keeps its token
    out: the chunks give numbers there, the walk's."""
    from binfer_b200.csrc import ops
    dev, T, H, d = cuda_device, 300, 2, 32
    torch.manual_seed(9)
    proj = torch.randn(T, 4 * H * d, device=dev).to(BF16)
    gates = torch.cat([torch.randn(T, H, device=dev),
                       torch.nn.functional.logsigmoid(2 + torch.randn(T, H, device=dev))], 1).contiguous()
    gates[[64, 100, 101, 299], H] = float("-inf")
    gates[[70, 128], 1] = float("-inf")
    qs = torch.tensor([0, T], dtype=torch.int32, device=dev)
    slots, err, outs = torch.zeros(1, dtype=torch.int32, device=dev), _err(dev), []
    for chunked in (False, True):
        out, state = torch.empty(T, H * d, device=dev), torch.zeros(
            1, H, ops.mlstm_state_size(d, d), device=dev)
        ops.mlstm_scan(proj, gates, state, qs, slots, out, 1, H, d, d, d ** -0.5, err, max_q=T,
                       chunked=chunked)
        outs.append(torch.cat([out.flatten(), state.flatten()]))
    assert bool(outs[0].isfinite().all())
    # as close as two orders of sums behind a quotient are (its denominator may be small)
    assert float((outs[1] - outs[0]).norm() / outs[0].norm()) <= 2e-5


@pytest.mark.parametrize("kind", ["linear", "delta", "mlstm", "retention"])
@pytest.mark.parametrize("own", [1, 70, 300])
def test_chunks_take_a_short_request_in_a_long_buffer(cuda_device, monkeypatch, kind, own):
    """One request that owns the first rows of a buffer long enough for chunks, nothing said about
    the longest portion: its rows are computed, the others left alone."""
    from binfer_b200.csrc import ops
    monkeypatch.setattr(ops, "DELTA_CHUNK_MIN", 160)
    dev, T, H, d = cuda_device, 300, 2, 32
    torch.manual_seed(8)
    qs = torch.tensor([0, own], dtype=torch.int32, device=dev)
    slots, err, outs = torch.zeros(1, dtype=torch.int32, device=dev), _err(dev), []
    x = torch.nn.functional.normalize(torch.randn(T, 2, H, d, device=dev), dim=-1)
    v, decay = torch.randn(T, H, d, device=dev), torch.rand(T, H, device=dev)
    flat = torch.cat([x.reshape(T, -1), v.reshape(T, -1)], 1).contiguous()
    for chunked in (False, True):
        out, state = torch.full((T, H * d), 7.0, device=dev), torch.zeros(1, H * d * d, device=dev)
        if kind == "linear":
            ops.linear_scan(x, v, decay, state, qs, slots, out, 1, H, H, d, d, err, chunked=chunked)
        elif kind == "delta":
            ops.delta_scan(flat, torch.stack([1 - decay, decay], 1).contiguous(), state, qs, slots,
                           out, 1, H, H, d, d, err, chunked=chunked)
        elif kind == "retention":
            ops.retention_scan(flat, 0, H * d, 2 * H * d, decay[0].contiguous(), None,
                               torch.arange(T, dtype=torch.int32, device=dev), state, qs, slots, out,
                               1, H, d, d, 1.0, err, chunked=chunked)
        else:
            state = torch.zeros(1, H, ops.mlstm_state_size(d, d), device=dev)
            ops.mlstm_scan(flat.to(BF16), torch.cat([decay, decay.log()], 1).contiguous(), state, qs,
                           slots, out, 1, H, d, d, 1.0, err, chunked=chunked)
        assert bool((out[own:] == 7.0).all())
        outs.append(torch.cat([out[:own].flatten(), state.flatten()]))
    _close(outs[1], outs[0], F32, scale=4)           # (sums of up to 300 terms, in other orders)


@pytest.mark.parametrize("kind", ["linear", "delta"])
def test_chunks_beside_many_single_tokens(cuda_device, kind):
    """A long portion has its chunks whatever else decodes in the step, and the same bits."""
    from binfer_b200.csrc import ops
    dev, n, singles, H, d = cuda_device, 400, 200, 64, 128
    torch.manual_seed(6)
    T, B, err, outs = n + singles, 1 + singles, _err(dev), []
    x = torch.nn.functional.normalize(torch.randn(T, 2, H, d, device=dev), dim=-1)
    v, decay = torch.randn(T, H, d, device=dev), torch.rand(T, H, device=dev)
    for t, b in ((T, B), (n, 1)):
        qs = torch.tensor([0] + list(range(n, t + 1)), dtype=torch.int32, device=dev)
        slots = torch.arange(b, dtype=torch.int32, device=dev)
        state, out = torch.zeros(b, H * d * d, device=dev), torch.empty(t, H * d, device=dev)
        before = ops.launches()
        if kind == "linear":
            ops.linear_scan(x[:t], v[:t], decay[:t], state, qs, slots, out, b, H, H, d, d, err,
                            max_q=n, chunked=True)
        else:
            qkv = torch.cat([x[:t].reshape(t, -1), v[:t].reshape(t, -1)], 1).contiguous()
            ops.delta_scan(qkv, torch.stack([1 - decay, decay], 1)[:t].contiguous(), state, qs,
                           slots, out, b, H, H, d, d, err, max_q=n, chunked=True)
        assert ops.launches() - before == 5 + (b > 1)    # (the walk serves the single tokens)
        outs.append((out[:n], state[0]))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("lens,H,dk,dv", [([161, 1, 192, 160, 257], 2, 24, 40),
                                          ([193], 3, 64, 100), ([320, 5], 1, 256, 64)])
def test_mlstm_scan_in_chunks(cuda_device, lens, H, dk, dv):
    """Against the walking kernel and both against float64: the products are no further off."""
    from binfer_b200.csrc import ops
    torch.manual_seed(len(lens) + dk)
    T, B, dev = sum(lens), len(lens), cuda_device
    proj = torch.randn(T, 2 * H * (dk + dv), device=dev).to(BF16)
    gates = torch.cat([2 * torch.randn(T, H, device=dev), torch.nn.functional.logsigmoid(
        3 + torch.randn(T, H, device=dev))], 1).contiguous()
    state = 0.1 * torch.randn(B + 1, H, ops.mlstm_state_size(dk, dv), device=dev)
    slots = torch.arange(B, dtype=torch.int32, device=dev).flip(0).contiguous()
    qs = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=dev)
    got, err = {}, _err(dev)
    for chunked in (False, True):
        s, o = state.clone(), torch.full((T, H * dv), 7.0, device=dev)
        ops.mlstm_scan(proj, gates, s, qs, slots, o, B, H, dk, dv, dk ** -0.5, err,
                       max_q=max(lens), chunked=chunked)
        got[chunked] = (o, s)
    assert int(err.item()) == 0 and torch.equal(got[True][1][B], state[B])
    off = {c: [0.0] * 4 for c in got}
    for b in range(B):
        a, e, at = int(qs[b]), int(qs[b + 1]), int(slots[b])
        x = proj[a:e].double()
        q = x[:, :H * dk].view(-1, H, dk) * dk ** -0.5
        k = x[:, H * dk:2 * H * dk].view(-1, H, dk)
        v = x[:, 2 * H * dk:2 * H * dk + H * dv].view(-1, H, dv)
        s0 = state[at].double()
        S, n, m = (s0[:, :dk * dv].view(H, dk, dv), s0[:, dk * dv:dk * dv + dk], s0[:, dk * dv + dk])
        o = torch.empty_like(v)
        for t in range(e - a):
            i, f = gates[a + t, :H].double(), gates[a + t, H:].double()
            m_new = torch.maximum(f + m, i)
            da, db = torch.exp(f + m - m_new), torch.exp(i - m_new)
            S = S * da[:, None, None] + (k[t] * db[:, None])[:, :, None] * v[t][:, None, :]
            n, m = da[:, None] * n + db[:, None] * k[t], m_new
            den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
            o[t] = (q[t][:, None, :] @ S)[:, 0] / den[:, None]
        for c, (go, gs) in got.items():
            g = gs[at].double()
            for i, (have, want) in enumerate((
                    (go[a:e].double().view(-1, H, dv), o), (g[:, :dk * dv].reshape(H, dk, dv), S),
                    (g[:, dk * dv:dk * dv + dk], n), (g[:, dk * dv + dk], m))):
                off[c][i] = max(off[c][i], float((have - want).norm() / want.norm()))
    for walk, products in zip(off[False], off[True]):
        assert products <= 1.5 * walk + 2e-7, off


# keys in whole steps of 64 and values in whole tiles of 128: the products on the tensor cores.  One chunk
# and its edges, chunks behind the 32 whose decays are at hand, one to three tiles of either, requests that
# are walked between them
@pytest.mark.parametrize("lens,H,dk,dv", [([161, 1, 192, 160, 257], 2, 64, 128), ([2177], 1, 64, 128),
                                          ([193, 320], 3, 128, 384), ([170, 3, 449], 2, 192, 256)])
def test_mlstm_chunks_on_tensor_cores(cuda_device, monkeypatch, lens, H, dk, dv):
    from binfer_b200.csrc import ops
    monkeypatch.setattr(ops, "MLSTM_TENSOR_MIN_CTAS", 0)
    test_mlstm_scan_in_chunks(cuda_device, lens, H, dk, dv)
    # rows off the 16-byte boundaries take the multiply-adds: the same but for the order of sums
    dev, T, B = cuda_device, sum(lens), len(lens)
    wide = torch.randn(T, 2 * H * (dk + dv) + 4, device=dev).to(BF16)
    gates = torch.cat([torch.randn(T, H, device=dev), -torch.rand(T, H, device=dev)], 1).contiguous()
    slots, err = torch.arange(B, dtype=torch.int32, device=dev), _err(dev)
    qs = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=dev)
    got = []
    for proj in (wide[:, 4:].contiguous(), wide[:, 4:]):
        s = torch.zeros(B, H, ops.mlstm_state_size(dk, dv), device=dev)
        o = torch.zeros(T, H * dv, device=dev)
        ops.mlstm_scan(proj, gates, s, qs, slots, o, B, H, dk, dv, dk ** -0.5, err, max_q=max(lens),
                       chunked=True)
        got.append((o, s))
    assert int(err.item()) == 0
    # (a request's outputs are quotients whose denominators may nearly vanish)
    assert float((got[0][0] - got[1][0]).norm() / got[1][0].norm()) < 2e-5
    assert float((got[0][1] - got[1][1]).norm() / got[1][1].norm()) < 1e-6
    bad = slots.clone()
    bad[0] = -1
    keep = got[0][1].clone()
    ops.mlstm_scan(wide[:, 4:].contiguous(), gates, keep, qs, bad, got[0][0], B, H, dk, dv, 1.0, err,
                   max_q=max(lens), chunked=True)
    assert int(err.item()) == 2 and torch.equal(keep[0], got[0][1][0])
    err.zero_()


@pytest.mark.parametrize("what", ["q", "k", "v"])
@pytest.mark.parametrize("at", [64, 140, 255])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_mlstm_chunks_on_tensor_cores_keep_infinities_apart(cuda_device, monkeypatch, what, at, bad):
    """What is not a number shows where the multiply-adds show it, and nowhere else changes a bit of the
    tokens before it and of the other head."""
    from binfer_b200.csrc import ops
    monkeypatch.setattr(ops, "MLSTM_TENSOR_MIN_CTAS", 0)
    dev, T, H, dk, dv = cuda_device, 300, 2, 128, 256
    torch.manual_seed(6)
    proj = torch.randn(T, 2 * H * (dk + dv), device=dev).to(BF16)
    gates = torch.cat([torch.randn(T, H, device=dev), -torch.rand(T, H, device=dev)], 1).contiguous()
    qs = torch.tensor([0, T], dtype=torch.int32, device=dev)
    slots, err, got = torch.zeros(1, dtype=torch.int32, device=dev), _err(dev), []
    column = {"q": dk + 5, "k": H * dk + dk + 5, "v": 2 * H * dk + dv + 130}[what]     # of head 1
    for spoil, walk in ((False, False), (True, False), (True, True)):
        x = proj.clone()
        if spoil:
            x[at, column] = bad
        s = torch.zeros(1, H, ops.mlstm_state_size(dk, dv), device=dev)
        o = torch.zeros(T, H * dv, device=dev)
        ops.mlstm_scan(x, gates, s, qs, slots, o, 1, H, dk, dv, dk ** -0.5, err, max_q=T, chunked=not walk)
        got.append((o.view(T, H, dv), s[0]))
    (clean, cs), (out, os), (want, ws) = got
    assert torch.equal(out[:, 0], clean[:, 0]) and torch.equal(os[0], cs[0])
    assert torch.equal(out[:at, 1], clean[:at, 1])
    assert torch.equal(out.isfinite(), want.isfinite()) and torch.equal(os.isfinite(), ws.isfinite())
    if what == "v":                                # (the other values' sizes)
        assert torch.equal(out[:, 1, :130], clean[:, 1, :130]) and torch.equal(out[:, 1, 131:], clean[:, 1, 131:])


def _mlstm_f64(proj, gates, s0, H, dk, dv, scale):
    """One request's outputs and last S, n, m in float64, token by token."""
    x = proj.double()
    q, k = x[:, :H * dk].view(-1, H, dk) * scale, x[:, H * dk:2 * H * dk].view(-1, H, dk)
    v = x[:, 2 * H * dk:2 * H * dk + H * dv].view(-1, H, dv)
    s0, g = s0.double(), gates.double()
    S, n, m = s0[:, :dk * dv].view(H, dk, dv), s0[:, dk * dv:dk * dv + dk], s0[:, dk * dv + dk]
    o = torch.empty_like(v)
    for t in range(x.shape[0]):
        m_new = torch.maximum(g[t, H:] + m, g[t, :H])
        da, db = torch.exp(g[t, H:] + m - m_new), torch.exp(g[t, :H] - m_new)
        S = S * da[:, None, None] + (k[t] * db[:, None])[:, :, None] * v[t][:, None, :]
        n, m = da[:, None] * n + db[:, None] * k[t], m_new
        den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
        o[t] = (q[t][:, None, :] @ S)[:, 0] / den[:, None]
    return o, S, n, m


# tiles by the hundred, so that a CTA goes from tile to tile (an even and an odd number of steps a tile),
# behind requests that are walked and, with a bad slot, past chunks that are left out
@pytest.mark.parametrize("dk,dv,H", [(64, 384, 6), (128, 512, 4), (192, 256, 8)])
@pytest.mark.parametrize("bad", [False, True])
def test_mlstm_chunks_on_tensor_cores_tile_after_tile(cuda_device, dk, dv, H, bad):
    """More than three tiles an SM, against float64 and no further off than the walking kernel."""
    from binfer_b200.csrc import ops
    dev, lens = cuda_device, [700, 1, 449, 30, 962, 161]
    torch.manual_seed(dk)
    T, B = sum(lens), len(lens)
    assert sum(-(-n // 64) for n in lens if n > 160) * H * (dv // 128) > 3 * 148
    proj = torch.randn(T, 2 * H * (dk + dv), device=dev).to(BF16)
    gates = torch.cat([2 * torch.randn(T, H, device=dev), torch.nn.functional.logsigmoid(
        3 + torch.randn(T, H, device=dev))], 1).contiguous()
    state = 0.1 * torch.randn(B + 1, H, ops.mlstm_state_size(dk, dv), device=dev)
    slots = torch.arange(B, dtype=torch.int32, device=dev).flip(0).contiguous()
    if bad:
        slots[2] = B + 1
    ends = [0] + list(torch.tensor(lens).cumsum(0))
    qs, err = torch.tensor(ends, dtype=torch.int32, device=dev), _err(dev)
    got = {}
    for chunked in (False, True):
        s, o = state.clone(), torch.full((T, H * dv), 7.0, device=dev)
        before = ops.launches()
        ops.mlstm_scan(proj, gates, s, qs, slots, o, B, H, dk, dv, dk ** -0.5, err, max_q=max(lens),
                       chunked=chunked)
        assert ops.launches() - before == (5 if chunked else 1)      # (four on the tensor cores, and the walk)
        assert int(err.item()) == (2 if bad else 0)
        err.zero_()
        got[chunked] = (o, s)
    for b in range(B):
        a, e, at = int(ends[b]), int(ends[b + 1]), int(slots[b])
        if bad and b == 2:
            assert bool((got[True][0][a:e] == 7.0).all())
            continue
        want = _mlstm_f64(proj[a:e], gates[a:e], state[at], H, dk, dv, dk ** -0.5)
        off = []
        for o, s in got.values():
            g = s[at].double()
            off.append([float((x - y).norm() / y.norm()) for x, y in zip(
                (o[a:e].double().view(-1, H, dv), g[:, :dk * dv].reshape(H, dk, dv),
                 g[:, dk * dv:dk * dv + dk], g[:, dk * dv + dk]), want)])
        for walk, products in zip(*off):
            assert products <= 1.5 * walk + 2e-7, (b, off)
    assert torch.equal(got[True][1][B], state[B])


# sizes and offsets that the tensor cores take; a key size, a value size and rows that they do not; few chunks
# of few heads and many; heads for the chip; single tokens beside a portion, which have no chunks
@pytest.mark.parametrize("T,H,dk,dv,off,singles,kernels", [
    (200, 2, 64, 128, 0, 0, 4), (200, 2, 256, 512, 8, 0, 4), (200, 2, 96, 128, 0, 0, 5), (200, 2, 64, 192, 0, 0, 5),
    (200, 2, 64, 128, 4, 0, 5), (319, 1, 64, 128, 0, 0, 4), (320, 39, 64, 128, 0, 0, 5), (320, 40, 64, 128, 0, 0, 4),
    (2000, 2, 256, 512, 0, 0, 5), (700, 3, 256, 512, 0, 0, 4), (700, 8, 128, 256, 0, 9, 5), (700, 8, 128, 256, 0, 0, 5)])
def test_mlstm_chunks_run_on_the_kernels_for_their_sizes(cuda_device, T, H, dk, dv, off, singles, kernels):
    """The kernels by name, as the profiler saw them, and their number, as the counter has it."""
    from binfer_b200.csrc import ops
    dev, B, n = cuda_device, 1 + singles, T
    T = T + singles
    proj = torch.randn(T, 2 * H * (dk + dv) + 8, device=dev).to(BF16)[:, off:off + 2 * H * (dk + dv)]
    gates = torch.cat([torch.randn(T, H, device=dev), -torch.rand(T, H, device=dev)], 1).contiguous()
    state = torch.zeros(B, H, ops.mlstm_state_size(dk, dv), device=dev)
    qs = torch.tensor([0] + list(range(n, T + 1)), dtype=torch.int32, device=dev)
    slots = torch.arange(B, dtype=torch.int32, device=dev)
    out, before = torch.empty(T, H * dv, device=dev), ops.launches()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        ops.mlstm_scan(proj, gates, state, qs, slots, out, B, H, dk, dv, dk ** -0.5, _err(dev), max_q=n,
                       chunked=True)
        torch.cuda.synchronize()
    assert ops.launches() - before == kernels + (B > 1)           # (the walk serves the single tokens)
    names = {n for e in prof.events() for n in ("mt_state", "mt_out", "cs_state", "cs_prefix", "cs_out")
             if n + "_kernel" in e.name}
    assert names == ({"mt_state", "mt_out"} if kernels == 4 else {"cs_state", "cs_prefix", "cs_out"}), names


# small and large: states, weighted values, weighted products of q and k, and bfloat16 numbers themselves
@pytest.mark.parametrize("what", ["values", "products", "keys", "queries", "large"])
def test_mlstm_chunks_on_tensor_cores_hold_floats_of_every_size(cuda_device, monkeypatch, what):
    """Nothing that multiply-adds over chunks hold is lost in terms: relative errors against float64, no
    further off.  (The walk is no measure: of keys or queries of 1e-39 its q . k are there in as many
    bits as they are multiplied, over chunks in those that a float of that size has.)"""
    from binfer_b200.csrc import ops
    monkeypatch.setattr(ops, "MLSTM_TENSOR_MIN_CTAS", 0)
    dev, T, H, dk, dv = cuda_device, 333, 2, 128, 256
    torch.manual_seed(9)
    size = {"values": (1, 1, 1e-35), "products": (1e-18, 1e-17, 1), "keys": (1, 1e-39, 1e28),
            "queries": (1e-39, 1, 1e28), "large": (1, 1, 1e33)}[what]
    x = torch.cat([c * torch.randn(T, n, device=dev) for c, n in zip(
        size, (H * dk, H * dk, H * dv))] + [torch.zeros(T, H * dv, device=dev)], 1).to(BF16)
    gates = torch.cat([2 * torch.randn(T, H, device=dev), torch.nn.functional.logsigmoid(
        3 + torch.randn(T, H, device=dev))], 1).contiguous()
    state = torch.randn(1, H, ops.mlstm_state_size(dk, dv), device=dev)
    state[:, :, :dk * dv] *= size[1] * size[2]
    state[:, :, dk * dv:dk * dv + dk] *= size[1]
    state[:, :, dk * dv + dk:] = 0.0
    qs = torch.tensor([0, T], dtype=torch.int32, device=dev)
    slots, err, off = torch.zeros(1, dtype=torch.int32, device=dev), _err(dev), []
    want = _mlstm_f64(x, gates, state[0], H, dk, dv, dk ** -0.5)
    for off16 in (4, 0):                       # (rows off the 16-byte boundaries: multiply-adds)
        proj = torch.zeros(T, x.shape[1] + 8, device=dev, dtype=BF16)[:, off16:off16 + x.shape[1]].copy_(x)
        s, o = state.clone(), torch.full((T, H * dv), 7.0, device=dev)
        ops.mlstm_scan(proj, gates, s, qs, slots, o, 1, H, dk, dv, dk ** -0.5, err, max_q=T, chunked=True)
        g = s[0].double()
        off.append([float((a - b).norm() / b.norm()) for a, b in zip(
            (o.double().view(-1, H, dv), g[:, :dk * dv].reshape(H, dk, dv),
             g[:, dk * dv:dk * dv + dk], g[:, dk * dv + dk]), want)])
    for adds, products in zip(*off):
        assert products <= 1.5 * adds + 2e-7, off


@pytest.mark.parametrize("at", [64, 140, 255])
@pytest.mark.parametrize("what", ["state", "q.k", "output", "faded"])
def test_mlstm_chunks_on_tensor_cores_with_products_that_overflow(cuda_device, monkeypatch, at, what):
    """Finite operands whose products leave float's range: the infinities and NaN of the multiply-adds."""
    from binfer_b200.csrc import ops
    monkeypatch.setattr(ops, "MLSTM_TENSOR_MIN_CTAS", 0)
    dev, T, H, dk, dv = cuda_device, 300, 2, 128, 256
    torch.manual_seed(6)
    wide = torch.randn(T, 2 * H * (dk + dv) + 4, device=dev).to(BF16)
    x = wide[:, 4:]
    q, k, v = x[:, dk:2 * dk], x[:, H * dk + dk:2 * H * dk], x[:, 2 * H * dk + dv:2 * H * dk + 2 * dv]   # of head 1
    if what == "state":
        k[at, 5], v[at, 130], v[at, 131] = 1.3e30, 1.7e30, -1.1e30
    elif what == "q.k":
        q[at, 5], k[at - 3, 5], v[at - 3, 130], v[at - 3, 131] = 1.3e18, 1.7e18, 1.1e30, -1.3e30
    elif what == "output":
        k[at - 20, 5], v[at - 20, 130], v[at - 20, 131], q[at, 5] = 1.3e15, 1.7e15, -1.1e15, 1.3e30
    else:                                      # (a state that the token's weight leaves out)
        at = at // 64 * 64
        k[at - 1, 5], v[at - 1, 130], v[at - 1, 131], q[at + 43, 5] = 1.3e15, 1.7e15, -1.1e15, 1.3e30
    gates = torch.cat([torch.randn(T, H, device=dev), -0.1 * torch.rand(T, H, device=dev)], 1).contiguous()
    if what == "faded":
        gates[:, H:] = -3.0
    qs = torch.tensor([0, T], dtype=torch.int32, device=dev)
    slots, err, got = torch.zeros(1, dtype=torch.int32, device=dev), _err(dev), []
    for proj in (x, x.contiguous()):           # (rows off the 16-byte boundaries: multiply-adds)
        s = torch.zeros(1, H, ops.mlstm_state_size(dk, dv), device=dev)
        o = torch.zeros(T, H * dv, device=dev)
        ops.mlstm_scan(proj, gates, s, qs, slots, o, 1, H, dk, dv, dk ** -0.5, err, max_q=T, chunked=True)
        got.append(torch.cat([o.flatten(), s.flatten()]))
    want, have = got
    assert bool(want.isfinite().all()) == (what == "faded")
    assert torch.equal(have.isnan(), want.isnan()) and torch.equal(have.isinf(), want.isinf())
    assert torch.equal(have[have.isinf()], want[have.isinf()])
    fin = want.isfinite()
    assert float((have - want)[fin].abs().max() / want[fin].abs().max()) < 1e-5


# ------------------------------------------- latent attention with keys and values expanded
# portions below, at and above a key tile of 64, a query tile of 128 and a block of 256, from the
# start and behind cached keys; the rows of two portions and a single token's row in one buffer
@pytest.mark.parametrize("portions,H,ps,sinks,gate", [
    ([(2, 0), (64, 63), (257, 130)], 3, 16, True, True), ([(128, 0), (130, 1)], 2, 8, False, False),
    ([(300, 500)], 1, 64, True, False), ([(65, 0)], 2, 16, False, True)])
def test_latent_attention_prefill_expanded(cuda_device, portions, H, ps, sinks, gate):
    from binfer_b200.csrc import ops
    torch.manual_seed(len(portions) + H)
    dev, rank, d, dr, dv = cuda_device, 32, 128, 64, 128
    ctx = [n + p for n, p in portions]
    T = 1 + sum(n for n, _ in portions)                  # the first row belongs to nobody here
    width = max(-(-c // ps) for c in ctx)
    n_pages = 1 + sum(-(-c // ps) for c in ctx)
    cache = torch.randn(n_pages, 1, ps, rank + dr, device=dev).to(BF16)
    order = torch.randperm(n_pages - 1) + 1              # pages anywhere in the pool
    tables = torch.full((len(ctx), width), -1, dtype=torch.int32)
    items, at, row = [], 0, 1
    for i, (n, p) in enumerate(portions):
        k = -(-ctx[i] // ps)
        tables[i, :k] = order[at:at + k]
        at += k
        items.append((i, row, n, p))
        row += n
    tables = tables.to(dev)
    items_d = torch.tensor(items, dtype=torch.int32, device=dev)
    rows = sum(-(-c // 64) * 64 for c in ctx)
    err = _err(dev)
    lat, rot, base = ops.latent_gather(cache, tables, items_d, len(items), rows, rank, err)
    w = (torch.randn(H * 256, rank, device=dev) * rank ** -0.5).to(BF16)
    kv = torch.mm(lat, w.t())
    wide = torch.randn(T, H * 192 + 8, device=dev).to(BF16)
    q = wide[:, 8:]                                      # a column block
    g = torch.randn(T, H + 3, device=dev).to(BF16)[:, 3:] if gate else None
    sk = torch.randn(H, device=dev) * 2 if sinks else None
    out = torch.full((T, H * 128 + 8), 7.0, device=dev, dtype=BF16)
    scale = 192 ** -0.5
    ops.latent_attention_prefill(q, kv, rot, base, items_d, len(items),
                                 max(n for n, _ in portions), out[:, 8:], H, scale, err, gate=g,
                                 sinks=sk)
    assert int(err.item()) == 0
    assert bool((out[:1] == 7).all()) and bool((out[:, :8] == 7).all())
    at = 0
    for i, (n, p) in enumerate(portions):
        assert int(base[i]) == at
        flat = cache[tables[i, :-(-ctx[i] // ps)].long(), 0].reshape(-1, rank + dr)[:ctx[i]]
        assert torch.equal(lat[at:at + ctx[i]], flat[:, :rank])
        assert torch.equal(rot[at:at + ctx[i]], flat[:, rank:])
        pad = -(-ctx[i] // 64) * 64
        assert float(lat[at + ctx[i]:at + pad].abs().sum() + rot[at + ctx[i]:at + pad].abs().sum()) == 0
        x = kv[at:at + ctx[i]].double().view(-1, H, 2, 128)
        k = torch.cat([x[:, :, 0], rot[at:at + ctx[i]].double()[:, None].expand(-1, H, -1)], -1)
        qq = q[items[i][1]:items[i][1] + n].double().view(n, H, 192)
        s = torch.einsum("qhd,khd->hqk", qq, k) * scale
        seen = torch.arange(ctx[i], device=dev)[None] <= torch.arange(p, p + n, device=dev)[:, None]
        s = s.masked_fill(~seen, -math.inf)
        if sinks:
            s = torch.cat([s, sk.double().view(H, 1, 1).expand(H, n, 1)], -1)
        o = torch.einsum("hqk,khd->qhd", torch.softmax(s, -1)[..., :ctx[i]], x[:, :, 1])
        if gate:
            o = o * torch.sigmoid(g[items[i][1]:items[i][1] + n].double())[:, :, None]
        have = out[items[i][1]:items[i][1] + n, 8:].double().view(n, H, 128)
        # probabilities and results are rounded to bfloat16 (2^-9 each)
        assert float((have - o).abs().max()) <= 2.0 ** -7 * float(o.abs().max()), i
        at += pad
    bad = tables.clone()
    bad[0, 0] = n_pages
    ops.latent_gather(cache, bad, items_d, len(items), rows, rank, err)
    assert int(err.item()) == 4
    err.zero_()


def test_latent_part_expands_portions_beside_single_tokens(cuda_device, monkeypatch):
    """A step of two portions and two single tokens, expanded and in latent coordinates."""
    from binfer_b200.config import FolivikConfig
    from binfer_b200.engine import StepItem, make_env, make_runner, model_from_seed
    from binfer_b200.parts import attention_latent
    cfg = FolivikConfig.from_dict({"vocab": 64, "width": 256, "norm": {"eps": 1e-5}, "layers": [
        {"type": "latent_attention", "mlp": None, "mixer": {
            "heads": 2, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 64, "q_rank": 96,
            "scale": 192 ** -0.5, "rot": {"base": 1e4, "dims": 64}}}]})
    env = make_env(BF16)
    model = model_from_seed(cfg, env, seed=3, std=0.06)
    runner = make_runner(model, env, page_size=16, num_pages=80, max_requests=4)
    mixer, view = model.blocks[0].mixer, runner.views[0]
    torch.manual_seed(5)
    lens = [(40, 150), (0, 70), (30, 1), (5, 1)]

    def one(expand):
        rule = (lambda self, q, out, ctx: sum(-(-c // 64) * 64 for n, c in zip(
            ctx.q_lens, ctx.ctx_lens_host) if n > 1)) if expand else (lambda *a: 0)
        monkeypatch.setattr(attention_latent.LatentAttention, "_expanded_rows", rule)
        torch.manual_seed(6)
        ys = []
        for i, (b, n) in enumerate(lens):
            runner.add_request(i)
            if b:
                x = torch.randn(b, 256, device=cuda_device).to(BF16)
                runner.reserve([StepItem(i, [0] * b)])
                ys.append(mixer.forward(x, runner.build_context([StepItem(i, [0] * b)]), view))
                runner.cache.commit(i, b)
        items = [StepItem(i, [0] * n) for i, (_, n) in enumerate(lens)]
        runner.reserve(items)
        x = torch.randn(sum(n for _, n in lens), 256, device=cuda_device).to(BF16)
        ys.append(mixer.forward(x, runner.build_context(items), view))
        for i in range(len(lens)):
            runner.free_request(i)
        runner.check_errors()
        return torch.cat(ys).double()

    plain, expanded = one(False), one(True)
    # both round what lies between the products to bfloat16, in other places
    assert float((plain - expanded).norm() / plain.norm()) <= 1.5e-2
    assert float((plain - expanded).abs().max()) <= 6e-2 * float(plain.abs().max())


@pytest.mark.parametrize("order", ["single tokens first", "portions first", "a short portion"])
def test_latent_part_chooses_and_splits_a_mixed_step(cuda_device, monkeypatch, order):
    """The part's own rule on a step of single tokens and a portion: a long portion is expanded and
    the single tokens in front of it are the only rows in latent coordinates, a short one is not."""
    from binfer_b200.config import FolivikConfig
    from binfer_b200.csrc import ops
    from binfer_b200.engine import StepItem, make_env, make_runner, model_from_seed
    H = 2
    cfg = FolivikConfig.from_dict({"vocab": 64, "width": 256, "norm": {"eps": 1e-5}, "layers": [
        {"type": "latent_attention", "mlp": None, "mixer": {
            "heads": H, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 64, "q_rank": 96,
            "scale": 192 ** -0.5, "rot": {"base": 1e4, "dims": 64}}}]})
    env = make_env(BF16)
    model = model_from_seed(cfg, env, seed=3, std=0.06)
    runner = make_runner(model, env, page_size=16, num_pages=120, max_requests=4)
    mixer, view = model.blocks[0].mixer, runner.views[0]
    long = 200 if order == "a short portion" else 1200
    lens = [(30, 1), (5, 1), (0, long)]
    if order == "portions first":
        lens = lens[::-1]
    calls = {"gather": 0, "rows": []}
    gather, attend = ops.latent_gather, ops.latent_attention

    def spy_gather(*a, **k):
        calls["gather"] += 1
        return gather(*a, **k)

    def spy_attend(q, *a, **k):
        calls["rows"].append(q.shape[0])
        return attend(q, *a, **k)
    monkeypatch.setattr(ops, "latent_gather", spy_gather)
    monkeypatch.setattr(ops, "latent_attention", spy_attend)

    def one(expands):
        mixer.expands = expands
        torch.manual_seed(6)
        for i, (b, n) in enumerate(lens):
            runner.add_request(i)
            if b:
                x = torch.randn(b, 256, device=cuda_device).to(BF16)
                runner.reserve([StepItem(i, [0] * b)])
                mixer.forward(x, runner.build_context([StepItem(i, [0] * b)]), view)
                runner.cache.commit(i, b)
        items = [StepItem(i, [0] * n) for i, (_, n) in enumerate(lens)]
        runner.reserve(items)
        x = torch.randn(sum(n for _, n in lens), 256, device=cuda_device).to(BF16)
        calls["gather"], calls["rows"] = 0, []
        y = mixer.forward(x, runner.build_context(items), view)
        for i in range(len(lens)):
            runner.free_request(i)
        runner.check_errors()
        return y.double(), calls["gather"], calls["rows"]

    plain, gathers, rows = one(False)
    assert gathers == 0 and rows == [long + 2]
    expanded, gathers, rows = one(True)
    if order == "a short portion":
        assert gathers == 0 and rows == [long + 2]
    else:
        assert gathers == 1 and rows == [2 if order == "single tokens first" else long + 2]
    assert float((plain - expanded).norm() / plain.norm()) <= 1.5e-2
    assert float((plain - expanded).abs().max()) <= 6e-2 * float(plain.abs().max())


# a window of one token, below, at and above a key tile and wider than some portions; kept tokens
# inside a tile, a whole tile, more than a tile and more than lies before the window; portions with
# cached keys; sinks alone with the keys shared out
@pytest.mark.parametrize("nh,nkv,ps,window,keep,sinks,splits", [
    (4, 2, 16, 64, 4, True, 1), (2, 2, 8, 1, 64, False, 1), (6, 2, 64, 200, 100, True, 1),
    (2, 1, 16, 90, 0, True, 1), (2, 1, 16, None, 0, True, 3)])
def test_prefill_attention_kept_tokens_and_sinks(cuda_device, nh, nkv, ps, window, keep, sinks,
                                                 splits):
    from binfer_b200.csrc import ops
    dev, d, gen = cuda_device, 128, torch.Generator().manual_seed(nh + ps + keep)
    ctxs, qlens = [300, 70, 700, 2, 257], [300, 37, 260, 2, 129]
    kcs, vcs, tables, qs, refs, items, base, row = [], [], [], [], [], [], 0, 0
    sk = torch.randn(nh, generator=gen) * 2 if sinks else None
    for b, (n, ql) in enumerate(zip(ctxs, qlens)):
        k = torch.randn(n, nkv, d, generator=gen).to(BF16).double()
        v = torch.randn(n, nkv, d, generator=gen).to(BF16).double()
        q = torch.randn(ql, nh, d, generator=gen).to(BF16).double()
        kh, vh = (x.repeat_interleave(nh // nkv, dim=1) for x in (k, v))
        sc = torch.einsum("qhd,nhd->hqn", q, kh) * d ** -0.5
        j, p = torch.arange(n)[None, :], (n - ql + torch.arange(ql))[:, None]
        seen = j <= p
        if window:
            seen = seen & ((p - j < window) | (j < keep))
        sc = sc.masked_fill(~seen[None], float("-inf"))
        if sinks:
            sc = torch.cat([sc, sk.double().view(nh, 1, 1).expand(nh, ql, 1)], -1)
        refs.append(torch.einsum("hqn,nhd->qhd", torch.softmax(sc, dim=-1)[..., :n], vh))
        kc, vc, ids = _paged(k, v, ps, "cpu", BF16, 70 + b, False)
        kcs.append(kc)
        vcs.append(vc)
        ids = [i + base for i in ids]
        if window:                       # pages that no query sees have been given back
            first = max(0, n - ql - window + 1) // ps
            ids = [i if x < -(-keep // ps) or x >= first else -1 for x, i in enumerate(ids)]
        tables.append(ids)
        base += kc.shape[0]
        qs.append(q)
        items.append([b, row, ql, n - ql])
        row += ql
    bt = torch.full((len(ctxs), max(len(t) for t in tables)), -1, dtype=torch.int32)
    for b, t in enumerate(tables):
        bt[b, :len(t)] = torch.tensor(t, dtype=torch.int32)
    q = torch.cat(qs).reshape(row, nh * d).to(BF16).to(dev)
    out, err = torch.zeros_like(q), _err(dev)
    ops.prefill_attention(q, torch.cat(kcs).to(dev), torch.cat(vcs).to(dev),
                          torch.tensor(items, dtype=torch.int32, device=dev), len(items), max(qlens),
                          bt.to(dev), out, nh, nkv, d, window, d ** -0.5, err, variant="umma2",
                          splits=splits, sinks=sk.to(dev) if sinks else None, keep_first=keep)
    assert int(err.item()) == 0
    _close(out.cpu(), torch.cat(refs).reshape(row, nh * d), BF16)


def test_split_prefill_on_two_streams_shares_no_scratch(cuda_device, monkeypatch):
    """The partial results of two calls on two streams lie in memory of their own."""
    from binfer_b200.csrc import ops
    nh, d, n, rows = 2, 128, 3000, 64
    q, kc, vc, sot, pos, bt, ref = _attention_case(cuda_device, BF16, nh, 1, d, 16, [n], [rows],
                                                   None, False, seed=31)
    items = torch.tensor([[0, 0, rows, n - rows]], dtype=torch.int32, device=cuda_device)
    real, spans = ops._run, []

    def spy(name, fn, *args):
        o, ml, splits = args[18].value, args[19].value, args[17].value
        size = rows * nh * splits * 4
        spans.extend([(o, o + size * d), (ml, ml + 2 * size)])
        real(name, fn, *args)
    monkeypatch.setattr(ops, "_run", spy)
    outs, err = [], _err(cuda_device)
    for _ in range(2):
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            outs.append(torch.zeros_like(q))
            ops.prefill_attention(q, kc, vc, items, 1, rows, bt, outs[-1], nh, 1, d, None, d ** -0.5,
                                  err, variant="umma2", max_ctx=n)
    torch.cuda.synchronize()
    spans.sort()
    assert len(spans) == 4 and all(a[1] <= b[0] for a, b in zip(spans, spans[1:]))
    for out in outs:
        _close(out, ref, BF16)


# ----------------------------------------------------------------- float32 attention in tiles
# rows below, at and above a tile of 64 and of 4, portions from the start and behind cached keys, a
# window inside, at and above a key tile
@pytest.mark.parametrize("nh,nkv,d,ps,window", [(4, 2, 128, 16, None), (3, 1, 64, 8, 64),
                                                (2, 2, 128, 64, 50), (8, 1, 64, 16, 200)])
def test_attention_f32_tiles(cuda_device, nh, nkv, d, ps, window):
    from binfer_b200.csrc import ops
    ctxs, qlens = [70, 200, 129, 300, 64, 1, 193], [70, 37, 5, 130, 64, 1, 1]
    q, kc, vc, sot, pos, bt, ref = _attention_case(cuda_device, F32, nh, nkv, d, ps, ctxs, qlens,
                                                   window, False, seed=21)
    qs = torch.tensor([0] + list(torch.tensor(qlens).cumsum(0)), dtype=torch.int32,
                      device=cuda_device)
    out, err = torch.full_like(q, 7.0), _err(cuda_device)
    ops.attention_f32(q, kc, vc, qs, pos, bt, out, len(ctxs), max(qlens), nh, nkv, d, window,
                      d ** -0.5, err)
    assert int(err.item()) == 0
    _close(out, ref, F32)
    # a row's bits do not depend on what shares its step: the last rows of every request alone
    # (tiles of four rows), each with its own table
    last = qs[1:].long() - 1
    one = torch.full((len(ctxs), nh * d), 7.0, device=cuda_device)
    each = torch.arange(len(ctxs) + 1, dtype=torch.int32, device=cuda_device)
    ops.attention_f32(q[last].contiguous(), kc, vc, each, pos[last].contiguous(), bt, one,
                      len(ctxs), 1, nh, nkv, d, window, d ** -0.5, err)
    assert torch.equal(one, out[last])
    # nor on the buffers that a context of one tile does without (a hint that is too small included)
    ops.attention_f32(q, kc, vc, qs, pos, bt, again := torch.full_like(q, 7.0), len(ctxs), max(qlens),
                      nh, nkv, d, window, d ** -0.5, err, max_ctx=64)
    assert torch.equal(again, out)
    bad = bt.clone()
    bad[0, 0] = kc.shape[0]
    ops.attention_f32(q, kc, vc, qs, pos, bad, out, len(ctxs), max(qlens), nh, nkv, d, window,
                      d ** -0.5, err)
    assert int(err.item()) == 4
    err.zero_()


# heads of 64 (two rows of a tile at a time) and of 128
@pytest.mark.parametrize("nh,nkv,d,window", [(8, 4, 128, None), (16, 8, 64, 70)])
def test_attention_f32_tiles_of_32_and_64_rows(cuda_device, nh, nkv, d, window):
    """Enough requests for an SM each take tiles of 64 rows, one request tiles of 32: the same bits."""
    from binfer_b200.csrc import ops
    ctxs = [33 + 17 * i for i in range(20)]
    qlens = [min(c, 40) for c in ctxs]
    q, kc, vc, sot, pos, bt, ref = _attention_case(cuda_device, F32, nh, nkv, d, 16, ctxs, qlens,
                                                   window, False, seed=22)
    ends = [0] + list(torch.tensor(qlens).cumsum(0))
    qs = torch.tensor(ends, dtype=torch.int32, device=cuda_device)
    out, err = torch.full_like(q, 7.0), _err(cuda_device)
    ops.attention_f32(q, kc, vc, qs, pos, bt, out, 20, 40, nh, nkv, d, window, d ** -0.5, err)
    assert int(err.item()) == 0
    _close(out, ref, F32)
    for b in (0, 7, 19):
        a, e = int(ends[b]), int(ends[b + 1])
        alone = torch.full((e - a, nh * d), 7.0, device=cuda_device)
        ops.attention_f32(q[a:e].contiguous(), kc, vc, torch.tensor([0, e - a], dtype=torch.int32,
                          device=cuda_device), pos[a:e].contiguous(), bt[b:b + 1].contiguous(), alone,
                          1, e - a, nh, nkv, d, window, d ** -0.5, err)
        assert torch.equal(alone, out[a:e])


@pytest.mark.parametrize("window", [None, 70])
def test_attention_f32_keys_that_a_row_does_not_see(cuda_device, window):
    """Values that are not finite reach the rows that see them alone; scores of -inf count as none.
    A portion's rows against the same rows alone, and against the kernel for any size."""
    from binfer_b200.csrc import ops
    n, at, d, dev = 200, 130, 64, cuda_device
    q, kc, vc, sot, pos, bt, ref = _attention_case(dev, F32, 2, 1, d, 16, [n], [n], window, False,
                                                   seed=22)
    def put(cache, key, x):
        cache[int(bt[0, key // 16]), 0, key % 16] = x
    put(vc, at, float("inf"))
    if window:
        put(vc, 3, float("nan"))
    q, err = q.abs(), _err(dev)
    for key in range(64):                # q . k overflows
        put(kc, key, -3e38)
    qs = torch.tensor([0, n], dtype=torch.int32, device=dev)
    out, want = torch.full_like(q, 7.0), torch.full_like(q, 7.0)
    ops.attention_f32(q, kc, vc, qs, pos, bt, out, 1, n, 2, 1, d, window, d ** -0.5, err)
    ops.paged_attention_generic(q, kc, vc, sot, pos, bt, want, 2, 1, d, window, d ** -0.5, err)
    fin = want.isfinite()
    assert torch.equal(fin, out.isfinite())
    # from the first key with a score on, or where the window has left the NaN behind
    assert bool(fin[73 if window else 64:at].all()) and not bool(fin[at:].any())
    assert not bool(fin[:64].any())
    one, each = torch.full_like(q[:1], 7.0), qs.new_tensor([0, 1])
    for t in (63, 64, 128, 129, 130, 199):
        ops.attention_f32(q[t:t + 1].contiguous(), kc, vc, each, pos[t:t + 1].contiguous(), bt, one,
                          1, 1, 2, 1, d, window, d ** -0.5, err)
        assert torch.equal(one[0].isfinite(), out[t].isfinite())
        assert torch.equal(one[0][one[0].isfinite()], out[t][out[t].isfinite()])
    assert int(err.item()) == 0
    _close(out[fin].cpu(), want[fin].cpu(), F32)


def _delta_on_tensor_cores(T, B, H, G, dk, dv):
    """Whether ``ops.delta_scan`` runs a step's chunks on the tensor cores: they take the sizes, and their scratch is
    within the limit."""
    from binfer_b200.csrc import ops
    fn = ops.lib().bf_chunk_scan_delta_scratch
    fn.restype = ops._c_ll
    return 0 < fn(*(ops._c_int(x) for x in (T, B, H, G, dk, dv, ops._chunk_limit(B, ops.DELTA_CHUNK_MIN), 1))) <= (
        ops.CHUNK_SCAN_MAX_BYTES)


@pytest.mark.parametrize("lens,H,G,dk,dv", [([161, 1, 192, 160, 257], 4, 2, 32, 24),
                                            ([300], 2, 1, 128, 128), ([193, 3], 3, 3, 68, 100),
                                            ([161, 1, 192, 160, 257], 4, 2, 128, 128),
                                            ([193, 320], 4, 2, 128, 64)])
def test_delta_scan_in_chunks(cuda_device, monkeypatch, lens, H, G, dk, dv):
    """Against the walking kernel and both against float64: the products are no further off."""
    from binfer_b200.csrc import ops
    monkeypatch.setattr(ops, "DELTA_CHUNK_MIN", 160)
    torch.manual_seed(len(lens) + dk)
    T, B, dev = sum(lens), len(lens), cuda_device
    assert _delta_on_tensor_cores(T, B, H, G, dk, dv) == (dk == 128)
    q, k = (torch.nn.functional.normalize(torch.randn(T, G, dk, device=dev), dim=-1)
            for _ in range(2))
    # neighbouring keys alike, so that a chunk's writes hang together
    k = torch.nn.functional.normalize(k + k.roll(1, 0), dim=-1)
    v = torch.randn(T, H, dv, device=dev)
    qkv = torch.cat([q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1)], 1).contiguous()
    gates = torch.rand(T, 2, H, device=dev)
    gates[:, 1] = 1 - 0.3 * gates[:, 1] ** 4
    gates[torch.rand(T, device=dev) < 0.02, 1] = 0.0
    state = torch.randn(B + 1, H * dk * dv, device=dev)
    slots = torch.arange(B, dtype=torch.int32, device=dev).flip(0).contiguous()
    qs = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=dev)
    got, err = {}, _err(dev)
    for chunked in (False, True):
        s, o = state.clone(), torch.full((T, H * dv), 7.0, device=dev)
        ops.delta_scan(qkv, gates, s, qs, slots, o, B, H, G, dk, dv, err, max_q=max(lens),
                       chunked=chunked)
        got[chunked] = (o, s)
    assert int(err.item()) == 0 and torch.equal(got[True][1][B], state[B])
    off = {c: [0.0] * 2 for c in got}
    for b in range(B):
        a, e, at = int(qs[b]), int(qs[b + 1]), int(slots[b])
        qd, kd = (x[a:e].double().repeat_interleave(H // G, 1) for x in (q, k))
        S = state[at].double().view(H, dv, dk).transpose(1, 2)
        want = torch.empty(e - a, H, dv, dtype=torch.float64, device=dev)
        for t in range(e - a):
            beta, g = gates[a + t].double()
            S = S * g[:, None, None]
            u = beta[:, None] * (v[a + t].double() - (kd[t][:, None, :] @ S)[:, 0])
            S = S + kd[t][:, :, None] * u[:, None, :]
            want[t] = (qd[t][:, None, :] @ S)[:, 0]
        for c, (go, gs) in got.items():
            have = gs[at].double().view(H, dv, dk).transpose(1, 2)
            for i, (x, y) in enumerate(((go[a:e].double().view(-1, H, dv), want), (have, S))):
                off[c][i] = max(off[c][i], float((x - y).norm() / y.norm()))
    for walk, products in zip(off[False], off[True]):
        assert products <= 1.5 * walk + 2e-7, off
    bad, keep = slots.clone(), got[True][1].clone()
    bad[0] = B + 5
    ops.delta_scan(qkv, gates, keep, qs, bad, o, B, H, G, dk, dv, err, max_q=max(lens), chunked=True)
    assert int(err.item()) == 2 and torch.equal(keep[int(slots[0])], got[True][1][int(slots[0])])
    err.zero_()


@pytest.mark.parametrize("what", ["v", "k", "q", "state"])
@pytest.mark.parametrize("dv", [64, 128])
def test_delta_chunks_keep_to_their_portion(cuda_device, monkeypatch, dv, what):
    """An infinity in the last of three portions, with a single token beside them: the numbers of that portion alone
    are not finite, the same ones as by multiply-adds, and the others' bits are the clean call's."""
    from binfer_b200.csrc import ops
    monkeypatch.setattr(ops, "DELTA_CHUNK_MIN", 160)
    lens, H, G, dk, dev = [193, 1, 320, 260], 4, 2, 128, cuda_device
    T, B, at = sum(lens), len(lens), sum(lens[:3]) + 70
    torch.manual_seed(17)
    q, k = (torch.nn.functional.normalize(torch.randn(T, G, dk, device=dev), dim=-1) for _ in range(2))
    v, s0 = torch.randn(T, H, dv, device=dev), torch.randn(B, H * dk * dv, device=dev)
    gates = torch.stack([torch.rand(T, H, device=dev), 1 - 0.05 * torch.rand(T, H, device=dev)], 1).contiguous()
    qs = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=dev)
    slots, err, got = torch.arange(B, dtype=torch.int32, device=dev), _err(dev), {}
    room = ops.CHUNK_SCAN_MAX_BYTES
    fn = ops.lib().bf_chunk_scan_delta_scratch
    fn.restype = ops._c_ll
    without = fn(*(ops._c_int(x) for x in (T, B, H, G, dk, dv, ops._chunk_limit(B, 160), 0)))
    for bad, tensor in ((False, True), (True, True), (True, False)):
        monkeypatch.setattr(ops, "CHUNK_SCAN_MAX_BYTES", room if tensor else without)
        assert _delta_on_tensor_cores(T, B, H, G, dk, dv) == tensor
        x = {"q": q.clone(), "k": k.clone(), "v": v.clone(), "state": s0.clone()}
        if bad:
            {"q": x["q"][at, 1], "k": x["k"][at, 0], "v": x["v"][at, 2], "state": x["state"][3]}[what][9] = math.inf
        qkv = torch.cat([x[n].reshape(T, -1) for n in "qkv"], 1).contiguous()
        o = torch.empty(T, H * dv, device=dev)
        ops.delta_scan(qkv, gates, x["state"], qs, slots, o, B, H, G, dk, dv, err, max_q=max(lens), chunked=True)
        got[bad, tensor] = (o, x["state"])
    assert int(err.item()) == 0
    (o0, clean), (o, s), (o_adds, s_adds) = got[False, True], got[True, True], got[True, False]
    assert bool(o0.isfinite().all()) and not bool(o.isfinite().all())
    assert torch.equal(o.isfinite(), o_adds.isfinite()) and torch.equal(s.isfinite(), s_adds.isfinite())
    assert torch.equal(o[:sum(lens[:3])], o0[:sum(lens[:3])]) and torch.equal(s[:3], clean[:3])


# keys at random, alike by a half and nearly the same; decays that forget in a few tokens and slow ones
@pytest.mark.parametrize("alike", [0.0, 0.5, 0.9])
@pytest.mark.parametrize("decays", ["fast", "slow"])
@pytest.mark.parametrize("kind", ["linear", "delta"])
def test_chunks_are_as_close_to_64_bits_as_the_walk(cuda_device, kind, decays, alike):
    """Relative errors over 777 tokens of 16 heads: a million numbers and more, so that what is left
    to chance is far below the tenth that is allowed."""
    from binfer_b200.csrc import ops
    T, H, d, dev = 777, 16, 128, cuda_device
    torch.manual_seed(13)
    norm = lambda x: torch.nn.functional.normalize(x, dim=-1)
    base = norm(torch.randn(H, d, device=dev))
    q = norm(torch.randn(T, H, d, device=dev))
    k = alike ** 0.5 * base + (1 - alike) ** 0.5 * norm(torch.randn(T, H, d, device=dev))
    v, g = torch.randn(T, H, d, device=dev), torch.rand(T, H, device=dev)
    if decays == "slow":
        g = 1 - 0.02 * g
    beta = torch.sigmoid(torch.randn(T, H, device=dev))
    s0 = 0.1 * torch.randn(1, H * d * d, device=dev)
    S, want = s0.double().view(H, d, d).transpose(1, 2), torch.empty(T, H, d, dtype=torch.float64,
                                                                       device=dev)
    qd, kd, vd, gd, bd = (x.double() for x in (q, k, v, g, beta))
    for t in range(T):
        S = S * gd[t][:, None, None]
        u = vd[t]
        if kind == "delta":
            u = bd[t][:, None] * (u - (kd[t][:, None] @ S)[:, 0])
        S = S + kd[t][:, :, None] * u[:, None]
        want[t] = (qd[t][:, None] @ S)[:, 0]
    qs = torch.tensor([0, T], dtype=torch.int32, device=dev)
    slots, err, off = torch.zeros(1, dtype=torch.int32, device=dev), _err(dev), []
    for chunked in (False, True):
        s, o = s0.clone(), torch.empty(T, H * d, device=dev)
        if kind == "linear":
            ops.linear_scan(torch.stack([q, k], 1).contiguous(), v, g, s, qs, slots, o, 1, H, H, d, d,
                            err, max_q=T, chunked=chunked)
        else:
            ops.delta_scan(torch.cat([x.reshape(T, -1) for x in (q, k, v)], 1).contiguous(),
                           torch.stack([beta, g], 1).contiguous(), s, qs, slots, o, 1, H, H, d, d,
                           err, max_q=T, chunked=chunked)
        have = s.double().view(H, d, d).transpose(1, 2)
        off.append([float((x - y).norm() / y.norm()) for x, y in ((o.double().view(T, H, d), want),
                                                                    (have, S))])
    # (or half a unit in the last place, which one rounding of the result is)
    for walk, products in zip(*off):
        assert products <= max(1.1 * walk, 2.0 ** -24), off


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("rest", [1, 15, 16, 17, 33, 48, 63])
def test_delta_chunks_weights_by_factors(cuda_device, rest, d):
    """A last chunk that ends at and beside each block of 16 tokens, decays of zero among slow ones (a
    factor of an earlier block is zero, or both of its sides are): relative errors of outputs and state
    against float64, beside the walk's 0.9 to 1.3e-7.  A chunk rounds the state once where the walk rounds it
    with every token: the products have 0.73 to 0.84 of the walk's errors with keys of 64 and 0.55 to 0.67 on the
    tensor cores, and weights that are half a unit in the last place off on one side would add more than is left."""
    from binfer_b200.csrc import ops
    T, H, dev = 7 * 64 + rest, 2, cuda_device
    torch.manual_seed(rest)
    q, k = (torch.nn.functional.normalize(torch.randn(T, H, d, device=dev), dim=-1) for _ in range(2))
    v, beta = torch.randn(T, H, d, device=dev), torch.rand(T, H, device=dev)
    g = (1 - 0.1 * torch.rand(T, H, device=dev)) * (torch.rand(T, H, device=dev) > 0.02)
    s0 = torch.randn(1, H * d * d, device=dev)
    S, want = s0.double().view(H, d, d).transpose(1, 2), []
    for qt, kt, vt, gt, bt in zip(*(x.double() for x in (q, k, v, g, beta))):
        S = S * gt[:, None, None]
        S = S + kt[:, :, None] * (bt[:, None] * (vt - (kt[:, None] @ S)[:, 0]))[:, None]
        want.append((qt[:, None] @ S)[:, 0])
    want, off = torch.stack(want), []
    qs = torch.tensor([0, T], dtype=torch.int32, device=dev)
    slots, err = torch.zeros(1, dtype=torch.int32, device=dev), _err(dev)
    for chunked in (False, True):
        s, o = s0.clone(), torch.empty(T, H * d, device=dev)
        ops.delta_scan(torch.cat([x.reshape(T, -1) for x in (q, k, v)], 1).contiguous(),
                       torch.stack([beta, g], 1).contiguous(), s, qs, slots, o, 1, H, H, d, d, err,
                       max_q=T, chunked=chunked)
        off.append([float((x - y).norm() / y.norm()) for x, y in
                    ((o.double().view(T, H, d), want), (s.double().view(H, d, d).transpose(1, 2), S))])
    for walk, products in zip(*off):
        assert products <= (0.75 if d == 128 else 0.9) * walk, off
    assert int(err.item()) == 0


@pytest.mark.parametrize("grows,first", [(60, 1e17), (84, 1e9)])
@pytest.mark.parametrize("kind,d", [("linear", 128), ("delta", 64), ("delta", 128)])
def test_chunks_of_decays_above_one(cuda_device, monkeypatch, kind, d, grows, first):
    """Twelve tokens of a block of 16 make the state e^grows times larger, thirty behind them e^100 times smaller:
    the tokens ahead of them (of values so large that they still count) have weights that are floats, one of whose
    two factors by the block's end is not, or without most of its bits.  (The delta rule's tokens between leave the
    state alone: its own u are of no use where weights leave the floats.)  Every token's result within the bound of
    its sums (d products of q and S, 64 weighted tokens, as many in u: 2^-24 each)."""
    from binfer_b200.csrc import ops
    T, H, dev = 500, 2, cuda_device
    torch.manual_seed(grows)
    q, k = (torch.nn.functional.normalize(torch.randn(T, H, d, device=dev), dim=-1) for _ in range(2))
    v, beta = 1e-30 * torch.randn(T, H, d, device=dev), torch.rand(T, H, device=dev)
    v[128:132] *= first
    beta[132:176] = 0.0
    g = 1 - 0.02 * torch.rand(T, H, device=dev)
    g[132:144], g[146:176] = math.exp(grows / 12), math.exp(-100 / 30)
    s0 = 1e-30 * torch.randn(1, H * d * d, device=dev)
    S, want = s0.double().view(H, d, d).transpose(1, 2), []
    for qt, kt, vt, gt, bt in zip(*(x.double() for x in (q, k, v, g, beta))):
        S = S * gt[:, None, None]
        u = bt[:, None] * (vt - (kt[:, None] @ S)[:, 0]) if kind == "delta" else vt
        S = S + kt[:, :, None] * u[:, None]
        want.append((qt[:, None] @ S)[:, 0])
    want = torch.stack(want)
    qs = torch.tensor([0, T], dtype=torch.int32, device=dev)
    slots, err = torch.zeros(1, dtype=torch.int32, device=dev), _err(dev)
    monkeypatch.setattr(ops, "LINEAR_TENSOR_MIN_CTAS", 0)
    s, o = s0.clone(), torch.empty(T, H * d, device=dev)
    if kind == "linear":
        qk = torch.stack([q, k], 1).contiguous()
        assert ops._chunk_scratch(True, T, T, 1, H, H, d, d, s, 0, qk, v, o)[1]
        ops.linear_scan(qk, v, g, s, qs, slots, o, 1, H, H, d, d, err, max_q=T, chunked=True)
    else:
        ops.delta_scan(torch.cat([x.reshape(T, -1) for x in (q, k, v)], 1).contiguous(),
                       torch.stack([beta, g], 1).contiguous(), s, qs, slots, o, 1, H, H, d, d, err,
                       max_q=T, chunked=True)
    c = (d + 128) * 2.0 ** -24
    off = (o.double().view(T, H, d) - want).norm(dim=2) / want.norm(dim=2)
    assert float(off.max()) <= c, (int(off.max(1)[0].argmax()), float(off.max()))
    assert float((s.double().view(H, d, d).transpose(1, 2) - S).norm() / S.norm()) <= c
    assert int(err.item()) == 0


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("taps", [1, 2, 3, 4])
@pytest.mark.parametrize("lens", [[1], [3, 1, 9, 2, 17], [1] * 5, [700, 1, 1, 643]])
def test_convolved_inputs_in_runs(cuda_device, lens, taps, dtype):
    """The encoders behind a short convolution, on rows of whole pieces of four (a thread takes a run
    of tokens) and on rows that are not (a warp per token): both against float64.  A sum of at most
    five products and a root mean square of 32 numbers keep float results within some 10 roundings;
    bfloat16 outputs are rounded once."""
    from binfer_b200.csrc import ops
    torch.manual_seed(len(lens) * 8 + taps)
    dev, T, B = cuda_device, sum(lens), len(lens)
    H, G, d, nh, nkv = 4, 2, 32, 4, 2
    C = (2 * G + H) * d                        # the same channels for all three encoders
    wide = torch.randn(T, C + 2 * H + 4, device=dev).to(dtype)
    odd = torch.empty(T, wide.shape[1] + 1, dtype=dtype, device=dev)[:, :-1]
    odd.copy_(wide)
    w, bias = torch.randn(C, taps, device=dev), torch.randn(C, device=dev)
    state = torch.randn(B + 1, max(1, (taps - 1) * C), device=dev)
    slots = torch.arange(B, dtype=torch.int32, device=dev).flip(0).contiguous()
    seq = torch.repeat_interleave(torch.arange(B), torch.tensor(lens)).int().to(dev)
    qs = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=dev)
    pos = torch.arange(T, dtype=torch.int32, device=dev)
    A_log, dt_bias, D = (torch.randn(H, device=dev) for _ in range(3))
    conv = torch.empty(T, C, dtype=torch.float64, device=dev)
    for b in range(B):
        a, e = int(qs[b]), int(qs[b + 1])
        u = torch.cat([state[int(slots[b])].double()[:(taps - 1) * C].view(taps - 1, C),
                       wide[a:e, :C].double()])
        conv[a:e] = sum(w[:, j].double() * u[j:j + e - a] for j in range(taps))
    softplus, silu = torch.nn.functional.softplus, torch.nn.functional.silu
    err, st = _err(dev), state if taps > 1 else None
    dt = softplus(wide[:, C:C + H].double() + dt_bias.double())
    pages, freqs = (T + 15) // 16, 1.0 / 10.0 ** (torch.arange(8, device=dev) / 8.0)
    for proj in (wide, odd):
        # the state space layer's
        qk, decay = torch.empty(T, 2, G, d, device=dev), torch.empty(T, H, device=dev)
        vf, skip = torch.empty(T, H, d, device=dev), torch.empty(T, H, d, device=dev)
        ops.mamba2_encode(proj, 0, C, w, bias, taps, st, slots, seq, qs, A_log, dt_bias, D, qk, vf,
                          skip, decay, H, G, d, d, err)
        y = silu(conv + bias.double())
        x = y[:, :H * d].view(T, H, d)
        _close(vf, x * dt[..., None], F32)
        _close(skip, x * D.double()[:, None], F32)
        _close(decay, torch.exp(-A_log.double().exp() * dt), F32)
        _close(qk[:, 1], y[:, H * d:H * d + G * d].view(T, G, d), F32)
        _close(qk[:, 0], y[:, H * d + G * d:].view(T, G, d), F32)
        # the delta rule's
        qkv, gates = torch.empty(T, C, device=dev), torch.empty(T, 2, H, device=dev)
        ops.delta_encode(proj, w, taps, st, slots, seq, qs, C + H, C, A_log, dt_bias, qkv, gates, H,
                         G, d, d, 1e-6, 0.25, err)
        y = silu(conv)
        q, k = y[:, :G * d].view(T, G, d), y[:, G * d:2 * G * d].view(T, G, d)
        unit = lambda z: z * torch.rsqrt((z * z).sum(-1, keepdim=True) + 1e-6)
        _close(qkv, torch.cat([unit(q).reshape(T, -1) * 0.25, unit(k).reshape(T, -1),
                               y[:, 2 * G * d:]], 1), F32, scale=4)
        _close(gates[:, 0], torch.sigmoid(wide[:, C + H:C + 2 * H].double()), F32)
        _close(gates[:, 1], torch.exp(-A_log.double().exp() * dt), F32)
        # attention's: heads of 32, 16 of them turned, divided by their root mean square
        q_out = torch.empty(T, nh * d, dtype=dtype, device=dev)
        kc = torch.zeros(pages, nkv, 16, d, dtype=dtype, device=dev)
        vc = torch.zeros_like(kc)
        ops.conv_encode(proj[:, :C], w, taps, st, slots, seq, qs, freqs, pos, pos, q_out, kc, vc, nh,
                        nkv, d, d, True, 1e-5, err)
        y = conv.view(T, nh + 2 * nkv, d).clone()
        ang = pos.double()[:, None, None] * freqs.double()
        lo, hi = y[:, :nh + nkv, :8].clone(), y[:, :nh + nkv, 8:16].clone()
        y[:, :nh + nkv, :8] = lo * ang.cos() - hi * ang.sin()
        y[:, :nh + nkv, 8:16] = hi * ang.cos() + lo * ang.sin()
        z = y[:, :nh + nkv]
        z = z * torch.rsqrt((z * z).mean(-1, keepdim=True) + 1e-5)
        flat = lambda c: c.transpose(1, 2).reshape(pages * 16, nkv, d)[:T]
        # (angles up to 1,343 in float: 2^-24 of the angle, beside the roundings)
        tol = 40 if dtype == F32 else 1
        _close(q_out.view(T, nh, d), z[:, :nh], dtype, scale=tol)
        _close(flat(kc), z[:, nh:], dtype, scale=tol)
        _close(flat(vc), y[:, nh + nkv:], dtype)
    assert int(err.item()) == 0


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("T,width,heads", [(1, 100, 1), (7, 2052, 8), (593, 1028, 9), (2, 50, 3)])
def test_mlstm_gates_tiles(cuda_device, T, width, heads, dtype):
    """Tiles of one and of four tokens, their remainders, and a width for the kernel of any size."""
    from binfer_b200.csrc import ops
    torch.manual_seed(T + width)
    h = torch.randn(T, width, device=cuda_device).to(dtype)
    w = (0.1 * torch.randn(2 * heads, width, device=cuda_device)).to(dtype)
    bias = torch.randn(2 * heads, device=cuda_device)
    gates = torch.empty(T, 2 * heads, device=cuda_device)
    ops.mlstm_gates(h, w, bias, gates, heads, 15.0)
    z = 15.0 * torch.tanh((h.double() @ w.double().T + bias.double()) / 15.0)
    z[:, heads:] = torch.nn.functional.logsigmoid(z[:, heads:])
    _close(gates, z, F32)


@pytest.mark.parametrize("what", ["weights", "state", "rows of states"])
def test_convolutions_off_a_boundary(cuda_device, what):
    """Weights, states or the way from state to state off 16-byte pieces: read as before."""
    from binfer_b200.csrc import ops
    torch.manual_seed(7)
    dev, T, H, G, d, taps = cuda_device, 5, 4, 2, 32, 4
    C = (H + 2 * G) * d
    proj = torch.randn(T, C + H, device=dev).to(BF16)
    w, bias = torch.randn(C, taps, device=dev), torch.randn(C, device=dev)
    state = torch.randn(2, (taps - 1) * C, device=dev)
    A_log, dt_bias, D = (torch.randn(H, device=dev) for _ in range(3))
    slots, qs = torch.tensor([1], dtype=torch.int32, device=dev), torch.tensor([0, T], dtype=torch.int32,
                                                                               device=dev)
    seq, err, got = torch.zeros(T, dtype=torch.int32, device=dev), _err(dev), []

    def off(x):
        y = torch.empty(x.numel() + 1, device=dev)[1:].view_as(x)
        return y.copy_(x)
    wide = torch.empty(2, state.shape[1] + 1, device=dev)
    for case in ("aligned", what):
        a = off(w) if case == "weights" else w
        b = off(state) if case == "state" else state
        if case == "rows of states":
            b = wide[:, :-1].copy_(state)
        qk, decay = torch.empty(T, 2, G, d, device=dev), torch.empty(T, H, device=dev)
        vf, skip = torch.empty(T, H, d, device=dev), torch.empty(T, H, d, device=dev)
        ops.mamba2_encode(proj, 0, C, a, bias, taps, b, slots, seq, qs, A_log, dt_bias, D, qk, vf,
                          skip, decay, H, G, d, d, err)
        got.append(torch.cat([x.flatten() for x in (qk, vf, skip, decay)]))
    assert int(err.item()) == 0
    _close(got[1], got[0], F32)


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("dv", [128, 256, 512, 1024, 96])
def test_head_norm_out_in_registers(cuda_device, dv, dtype):
    """The sizes whose numbers stay in registers and one that does not, rows of odd offsets too."""
    from binfer_b200.csrc import ops
    torch.manual_seed(dv)
    T, H, dev = 5, 3, cuda_device
    o, skip = torch.randn(T, H * dv, device=dev), torch.randn(T, H * dv, device=dev)
    w = torch.randn(H * dv, device=dev)
    proj = torch.randn(T, H * dv + 12, device=dev).to(dtype)
    for off in (8, 7):
        g = torch.nn.functional.silu(proj[:, off:off + H * dv].double()).view(T, H, dv)
        sg = torch.sigmoid(proj[:, off:off + H * dv].double()).view(T, H, dv)
        rms = lambda x: x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-5)
        x, wd = o.double().view(T, H, dv), w.double().view(H, dv)
        out = torch.empty(T, H * dv, dtype=dtype, device=dev)
        ops.gate_norm_out(o, skip, proj, off, w, out, H, 1e-5)
        _close(out.view(T, H, dv), rms((x + skip.double().view(T, H, dv)) * g) * wd, dtype)
        ops.mlstm_out(o, proj, off, w, out, H, dv, 1e-5)
        _close(out.view(T, H, dv), rms(x) * wd * sg, dtype)
        ops.retention_out(o, proj, off, out, H, dv, 1e-5)
        _close(out.view(T, H, dv), rms(x) * g, dtype)


@pytest.mark.parametrize("T,width,E,ff,ff_sh,top,ident,gate,kind", [
    (1, 64, 1, 8, 0, 1, 0, False, "silu"), (257, 192, 5, 72, 40, 2, 0, True, "clamped"),
    (700, 128, 3, 128, 0, 2, 4, False, "silu"), (1500, 256, 64, 64, 264, 3, 0, False, "silu"),
    (300, 136, 8, 32, 8, 8, 2, True, "silu")])
def test_moe_grouped(cuda_device, T, width, E, ff, ff_sh, top, ident, gate, kind):
    """Chosen experts alone against float64 from the same bfloat16 numbers.  The activations are
    rounded to bfloat16 once, their float sums once: 2^-8 of the largest magnitude each at most."""
    from binfer_b200.csrc import ops
    torch.manual_seed(T + E)
    dev, F = cuda_device, E * ff + ff_sh
    h = torch.randn(T, width + 8, device=dev).to(BF16)[:, :width]
    gu = (torch.randn(2 * F, width, device=dev) * width ** -0.5).to(BF16)
    down = (torch.randn(width, F, device=dev) * ff ** -0.5).to(BF16)
    ids = torch.stack([torch.randperm(E + ident)[:top] for _ in range(T)])
    if E > 4:                                    # an expert that nobody chose, and one for all
        ids[ids == 1] = 0
        ids[:, 0] = 2
    ids = ids.to(dev, torch.int32).contiguous()
    tw = torch.rand(T, top, device=dev)
    cols = E + gate + (ident > 0)
    rw = torch.rand(T, cols, device=dev)
    act = ops.ExpertAct(kind, 1.0, 0.7, 1.3, 0.5)
    out, err = torch.full((T, width), 7.0, dtype=BF16, device=dev), ops.error_word(dev)
    ops.moe_grouped(h, gu, down, ids, tw, rw, out, E, ff, ff_sh, top, shared_gate=gate,
                    identity_col=cols - 1 if ident else -1, expert_act=act)
    x, g = h.double(), gu.double()

    def run(lo, n, limit):
        a, u = x @ g[lo:lo + n].T, x @ g[F + lo:F + lo + n].T
        if kind == "clamped":
            a, u = a.clamp(max=limit), u.clamp(-limit, limit) + 0.5
        z = a * torch.sigmoid((1.3 if kind == "clamped" else 1.0) * a) * u
        return z, down[:, lo:lo + n].double().T
    ref = torch.zeros(T, width, dtype=torch.float64, device=dev)
    for e in range(E):
        z, d = run(e * ff, ff, 1.0)
        for j in range(top):
            ref += torch.where((ids[:, j] == e)[:, None], tw[:, j:j + 1].double() * (z @ d), 0.0)
    if ff_sh:
        z, d = run(E * ff, ff_sh, 0.7)
        ref += (rw[:, E:E + 1].double() if gate else 1.0) * (z @ d)
    if ident:
        ref += rw[:, -1:].double() * x
    assert int(err.item()) == 0
    _close(out, ref, BF16)


@pytest.mark.parametrize("identity,shared,gate", [(2, 64, True), (0, 0, False)])
def test_moe_part_takes_the_chosen_experts_alone(cuda_device, monkeypatch, identity, shared, gate):
    """The part's own rule and what it hands over, against every expert for every token; a column
    block that the grouped kernels cannot read stays there."""
    from binfer_b200.config import MoESpec
    from binfer_b200.csrc import ops
    from binfer_b200.engine import make_env
    from binfer_b200.parts import moe
    dev, T, width, E = cuda_device, 1100, 256, 8
    spec = MoESpec(num_experts=E, top=2, expert_size=64, shared_size=shared, shared_gate=gate,
                   identity=identity, scoring="softmax_all" if identity else "softmax_top")
    part = moe.MoEFeedForward(spec, width, "", make_env(BF16))
    torch.manual_seed(12)
    part.load(lambda s: (torch.randn(s.shape, device=dev) * s.shape[-1] ** -0.5).to(
        F32 if s.role == "vector" else BF16))
    wide = torch.randn(T, width + 8, device=dev).to(BF16)
    x, calls, grouped = wide[:, :width].contiguous(), [], ops.moe_grouped
    monkeypatch.setattr(ops, "moe_grouped", lambda *a, **k: (calls.append(1), grouped(*a, **k)))
    every = part.forward(x, None).double()                   # (far fewer operations than the rule's)
    assert not calls
    monkeypatch.setattr(moe, "GROUPED_MIN_FLOPS", 1)
    chosen = part.forward(x, None).double()
    assert len(calls) == 1
    # activations rounded to bfloat16 and results rounded once on either side
    assert float((chosen - every).norm() / every.norm()) <= 1e-2
    assert float((chosen - every).abs().max()) <= 2.0 ** -6 * float(every.abs().max())
    wide[:, 1:1 + width] = x
    apart = part.forward(wide[:, 1:1 + width], None).double()
    assert len(calls) == 1 and float((apart - every).norm() / every.norm()) <= 1e-2
    monkeypatch.setattr(moe, "GROUPED", False)
    part.forward(x, None)
    assert len(calls) == 1
