"""Sizes at which a launch changes its shape: decode spans and page tables among the kernel arguments, clusters and head pairs
of the backward, the polynomial exponent of head_dim 64, ALiBi slopes among the kernel arguments."""
import numpy as np
import pytest
import torch

from oracle import binding as ob
from tests.gpu_util import bf16_round, ctx, dev, fa, run_forward
from tests.test_gpu_backward_bf16 import randn
from tests.test_gpu_chunked_backward import run_backward
from tests.test_gpu_decode_cache import oracle_decode, run_batched, unpack

pytestmark = pytest.mark.gpu


# tokens and page size: clusters around one tile and at their longest (4096 tokens, 256 pages, the largest table that travels
# with the launch); spans with a table in memory, and with one that travels: longer contexts in larger pages, more KV heads than
# clusters take
@pytest.mark.parametrize("n,page", [(1, 16), (15, 16), (16, 16), (17, 16), (33, 16), (256 * 16, 16), (256 * 16 + 1, 16), (4097, 32),
                                    (8192, 32), (8193, 32), (6145, 64)])
@pytest.mark.parametrize("Hq,Hkv,D", [(8, 2, 64), (32, 8, 128), (16, 16, 128)])
def test_paged_decode_spans_and_tables(n, page, Hq, Hkv, D):
    c = ctx()
    cache = fa.CudaPagedKvCache(c, fa.BF16, page, (n + page - 1) // page + 1, Hkv, D)
    g = torch.Generator().manual_seed(n)
    k, v, q = (torch.randn(r * D, generator=g).bfloat16() for r in (n * Hkv, n * Hkv, Hq))
    cache.record_append(k.cuda(), v.cuda(), n)
    out = c.create_decode_output_buffer(fa.BF16, 1, Hq, D)
    out.fill_(0x7f)
    before = c.launch_count()
    c.decode_paged(fa.BF16, cache.table(), Hq, Hkv, D, fa.config(True), 5e5, n - 1, q.cuda(), cache.k_buffer(), cache.v_buffer(), out)
    assert c.launch_count() - before == (1 if n <= (2048 if Hkv == 16 else 4096) else 2)  # a cluster, or spans and a merge
    o, l = unpack(out, fa.BF16, Hq, D)
    eo, el = oracle_decode(q.float().numpy(), k.float().numpy().reshape(n, -1), v.float().numpy().reshape(n, -1), Hq, Hkv, D, 5e5,
                           n - 1, 0, True)
    assert np.abs(o.reshape(-1) - eo.reshape(-1)).max() <= 2e-2
    assert np.abs(l.reshape(-1) - el.reshape(-1)).max() <= 2e-3
    assert c.device_status() == 0


# lengths of the batch: single sequences on either side of the span rule, a full batch of short ones, and one long among many
# short ones, whose parts (dense over all sequences) would take four times the memory with spans of 16 tokens
@pytest.mark.parametrize("lens", [[4097], [6144], [6145], [6000], [8000], [700] * 16, [700] * 20, [100] * 128, [2048] + [16] * 18,
                                  [2048] + [16] * 127, [2064] + [16] * 18])
def test_decode_asks_for_no_more_workspace_than_spans_of_64(lens):
    """Shorter spans keep their parts in memory of the context: the workspace is bounded by the parts of 64-token spans."""
    Hq, Hkv, D, page, c = 32, 8, 128, 16, fa.Context(0)
    pages = [-(-n // page) for n in lens]
    g = torch.Generator().manual_seed(3)
    Q = torch.randn(len(lens), Hq * D, generator=g).bfloat16()
    K, V = (torch.randn(sum(pages) * page, Hkv * D, generator=g).bfloat16() for _ in range(2))
    tables = np.zeros((len(lens), max(pages)), np.int32)
    for i, n in enumerate(pages):
        tables[i, :n] = sum(pages[:i]) + np.arange(n)
    args = (fa.BF16, np.array(lens, np.int32), tables, sum(pages), max(pages), Q, K, V, Hq, Hkv, D, page, 5e5)
    o, l = run_batched(c, *args)
    assert c.launch_count() == 2  # spans and a merge, not a cluster
    padded = [-(-n // 16) * 16 for n in lens]
    span = max(64, (-(-sum(padded) // (2 * 148)) + 15) // 16 * 16)
    parts = -(-max(padded) // span) + 1
    assert c.workspace_bytes() <= (1 << 16) + parts * len(lens) * Hq * (D + 1) * 4 + 256
    eo, el = run_batched(ctx(), *args, splits=1)
    assert np.abs(o - eo).max() <= 2e-2 and np.abs(l - el).max() <= 2e-3
    assert c.device_status() == 0


# lengths around the cluster sizes of short contexts (128 tokens per CTA with one tile per warp, eight CTAs, four tiles per
# warp), mixed batches whose shortest sequence leaves warps and CTAs without a token, and one sequence more than SMs allow
@pytest.mark.parametrize("lens", [[128], [129], [513], [1024], [1025], [4096], [4097], [1, 17, 900], [2000, 3, 129, 64], [300] * 18,
                                  [300] * 19])
@pytest.mark.parametrize("Hq,Hkv,D", [(8, 8, 64), (32, 8, 128), (64, 8, 128)])
def test_decode_clusters(lens, Hq, Hkv, D):
    """Against the same call with one part per sequence (P is rounded to bf16, 2^-9, relative to another running maximum)."""
    page, c = 16, ctx()
    pages = [-(-n // page) for n in lens]
    g = torch.Generator().manual_seed(7)
    Q = torch.randn(len(lens), Hq * D, generator=g).bfloat16()
    K, V = (torch.randn(sum(pages) * page, Hkv * D, generator=g).bfloat16() for _ in range(2))
    tables = np.zeros((len(lens), max(pages)), np.int32)
    order = np.random.default_rng(1).permutation(sum(pages))
    for i, n in enumerate(pages):
        tables[i, :n] = order[sum(pages[:i]):sum(pages[:i]) + n]
    args = (fa.BF16, np.array(lens, np.int32), tables, sum(pages), max(pages), Q, K, V, Hq, Hkv, D, page, 5e5)
    o, l = run_batched(c, *args)
    eo, el = run_batched(c, *args, splits=1)
    assert np.abs(o - eo).max() <= 2e-2 and np.abs(l - el).max() <= 2e-3
    again, al = run_batched(c, *args)
    assert np.array_equal(o, again) and np.array_equal(l, al)
    assert c.device_status() == 0


@pytest.mark.parametrize("lens,at", [([40], [(0, 1)]), ([40, 16], [(1, 0)]), ([900, 700], [(0, 0), (0, 40), (1, 43)])])
def test_decode_clusters_skip_pages_outside_the_pool(lens, at):
    """Entries of the device's page table that are outside the pool are not read: their tokens count for nothing, a sequence
    without any other gets O = 0 and LSE = -inf, and the call is flagged."""
    Hq, Hkv, D, page, c = 8, 2, 64, 16, ctx()
    pages = [-(-n // page) for n in lens]
    g = torch.Generator().manual_seed(11)
    Q = torch.randn(len(lens), Hq * D, generator=g).bfloat16()
    K, V = (torch.randn(sum(pages) * page, Hkv * D, generator=g).bfloat16() for _ in range(2))
    tables = np.zeros((len(lens), max(pages)), np.int32)
    for i, n in enumerate(pages):
        tables[i, :n] = sum(pages[:i]) + np.arange(n)
    broken, qpos = tables.copy(), np.array(lens, np.int32) - 1
    for k, (s, i) in enumerate(at):
        broken[s, i] = -1 if k % 2 else sum(pages) + 1000
    out = c.create_decode_output_buffer(fa.BF16, len(lens), Hq, D)
    before = c.launch_count()
    c.decode_paged_batched(fa.BF16, len(lens), Hq, Hkv, D, page, sum(pages), max(pages), *(torch.from_numpy(x).cuda() for x in
                           (broken, np.array(lens, np.int32), qpos)), tables, np.array(lens, np.int32), qpos, fa.config(True), 5e5,
                           Q.cuda(), K.cuda(), V.cuda(), out)
    assert c.launch_count() - before == 1
    assert c.device_status() == 35  # FLAT_ERR_PAGE_OUT_OF_RANGE, cleared by the read
    o, l = unpack(out, fa.BF16, len(lens) * Hq, D)
    o, l = o.reshape(len(lens), Hq, D), l.reshape(len(lens), Hq)
    for s, n in enumerate(lens):
        rows = [tables[s, t // page] * page + t % page for t in range(n) if (s, t // page) not in at]
        if not rows:
            assert not o[s].any() and np.isneginf(l[s]).all()
            continue
        eo, el = oracle_decode(Q[s].float().numpy(), K.float().numpy()[rows], V.float().numpy()[rows], Hq, Hkv, D, 5e5, n - 1, 0, True)
        assert np.abs(o[s].reshape(-1) - eo.reshape(-1)).max() <= 2e-2
        assert np.abs(l[s].reshape(-1) - el.reshape(-1)).max() <= 2e-3


# tokens: clusters of one CTA and of eight (one tile per warp, several), and spans with a merge
@pytest.mark.parametrize("n", [10, 40, 700, 4096, 6000])
def test_decode_of_scores_that_are_not_finite(n):
    """A NaN in a query, or in a key, reaches O of the heads that meet it, whichever warp or CTA has the key; the other heads keep
    every bit.  Keys whose score overflows to -inf count for nothing."""
    Hq, Hkv, D, page, c = 8, 2, 128, 16, ctx()
    G = Hq // Hkv
    rng = torch.Generator().manual_seed(n)
    k, v = (torch.randn(n, Hkv, D, generator=rng).bfloat16() for _ in range(2))
    q = torch.randn(Hq, D, generator=rng).bfloat16()

    def decode(q, k):
        cache = fa.CudaPagedKvCache(c, fa.BF16, page, -(-n // page), Hkv, D)
        cache.record_append(k.reshape(-1).cuda(), v.reshape(-1).cuda(), n)
        out = c.create_decode_output_buffer(fa.BF16, 1, Hq, D)
        before = c.launch_count()
        c.decode_paged(fa.BF16, cache.table(), Hq, Hkv, D, fa.config(True), 5e5, n - 1, q.reshape(-1).cuda(), cache.k_buffer(),
                       cache.v_buffer(), out)
        assert c.launch_count() - before == (1 if n <= 4096 else 2)  # a cluster, or spans and a merge
        return unpack(out, fa.BF16, Hq, D)

    o, l = (x.reshape(Hq, -1) for x in decode(q, k))
    bad = q.clone()
    bad[1, 5] = float("nan")
    bo, bl = (x.reshape(Hq, -1) for x in decode(bad, k))
    others = np.arange(Hq) != 1
    assert np.isnan(bo[1]).all() and not np.isfinite(bl[1]).any()
    assert np.array_equal(bo[others], o[others]) and np.array_equal(bl[others], l[others])
    for token in (0, n // 2, n - 1):
        bad = k.clone()
        bad[token, 1, 5] = float("nan")
        bo, bl = (x.reshape(Hq, -1) for x in decode(q, bad))
        assert np.isnan(bo[G:]).all(), token
        assert np.isnan(bl[G:]).all() or n > 4096, token
        assert np.array_equal(bo[:G], o[:G]) and np.array_equal(bl[:G], l[:G]), token
    # The last pair of dimensions turns by at most 6000 * 5e5^(-126/128) = 0.015, and Q is scaled by 2^-3: 2^64 against -2^70
    # overflows, but not the low half of Q (2^-8 of it at most) against it.  The other tokens' k there is 0.
    big, low = q.clone(), k.clone()
    big[0] = 0
    big[0, 126] = 2.0 ** 64
    low[:, 0, 126:] = 0
    low[:min(n - 1, 100), 0, 126] = -2.0 ** 70
    bo, bl = (x.reshape(Hq, -1) for x in decode(big, low))
    live = n - min(n - 1, 100)
    assert np.abs(bo[0] - v[-live:, 0].float().mean(0).numpy()).max() <= 2e-2
    assert abs(bl[0, 0] - np.log(live)) <= 2e-3
    assert c.device_status() == 0


# (B, Hq, Hkv, N, D): clusters of 1, 4, 3, 8 and 8 CTAs per key tile on 148 SMs, with and without a mask
@pytest.mark.parametrize("B,Hq,Hkv,N,D", [(1, 4, 4, 100, 64), (1, 8, 1, 130, 128), (1, 12, 1, 128, 64), (1, 32, 2, 600, 64),
                                          (1, 16, 1, 700, 128)])
@pytest.mark.parametrize("causal", [True, False])
def test_backward_clusters(B, Hq, Hkv, N, D, causal):
    q, k, v, do = randn(B * Hq * N * D, 1), randn(B * Hkv * N * D, 2), randn(B * Hkv * N * D, 3), randn(B * Hq * N * D, 4)
    fo, fl = run_forward("grouped", fa.F32, fa.shape(B, Hq, Hkv, N, N, D), fa.config(causal), q, k, v)
    fo = bf16_round(fo)
    got = run_backward(fa.BF16, B, Hq, Hkv, N, D, causal, None, q, k, v, do, fo, fl)
    exp = run_backward(fa.F32, B, Hq, Hkv, N, D, causal, None, q, k, v, do, fo, fl)
    for name, a, e in zip(("dQ", "dK", "dV"), got, exp):
        # P and dS are rounded to bf16 (2^-9) before a sum of N * group terms of mixed sign: 2e-2 holds for the small sums of
        # the other backward tests, here it grows with the largest gradient
        assert np.abs(a - e).max() <= 2e-2 + 4e-3 * np.abs(e).max(), (name, float(np.abs(a - e).max()), float(np.abs(e).max()))
    again = run_backward(fa.BF16, B, Hq, Hkv, N, D, causal, None, q, k, v, do, fo, fl)
    assert all(np.array_equal(x, y) for x, y in zip(got, again))
    assert ctx().device_status() == 0


def cluster_and_fewest_pairs(B, Hq, Hkv, N, causal, sms=148):
    """CTAs per key tile as the launch chooses them, and the (head, query tile) pairs of the key tile that has the fewest."""
    n, group = -(-N // 128), Hq // Hkv
    pairs, longest = (n * (n + 1) // 2 if causal else n * n) * Hq * B, n * group
    parts = 1
    while parts < 8 and (parts + 1) * 4 <= longest and 4 * (-(-longest // parts)) * sms > 5 * pairs:
        parts += 1
    return parts, group if causal else longest


# the last key tile has 1 pair for 2 CTAs, 4 for 8
@pytest.mark.parametrize("Hq,Hkv,N,parts", [(16, 16, 1000, 2), (8, 2, 1500, 8)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("budget", [0, 8 << 30])
def test_backward_clusters_with_idle_ctas(Hq, Hkv, N, parts, D, budget):
    """CTAs of a cluster without a pair of their own: they stream nothing and still add their share of the others' sums."""
    size, fewest = cluster_and_fewest_pairs(1, Hq, Hkv, N, True)
    assert size == parts and fewest < size
    q, k, v, do = randn(Hq * N * D, 11), randn(Hkv * N * D, 12), randn(Hkv * N * D, 13), randn(Hq * N * D, 14)
    fo, fl = run_forward("grouped", fa.F32, fa.shape(1, Hq, Hkv, N, N, D), fa.config(True), q, k, v)
    fo = bf16_round(fo)
    exp = run_backward(fa.F32, 1, Hq, Hkv, N, D, True, None, q, k, v, do, fo, fl)
    ctx().set_backward_scratch_budget(budget)
    try:
        got, again = (run_backward(fa.BF16, 1, Hq, Hkv, N, D, True, None, q, k, v, do, fo, fl) for _ in range(2))
    finally:
        ctx().set_backward_scratch_budget(8 << 30)
    for name, a, e in zip(("dQ", "dK", "dV"), got, exp):  # the bound of the test above
        assert np.abs(a - e).max() <= 2e-2 + 4e-3 * np.abs(e).max(), (name, float(np.abs(a - e).max()), float(np.abs(e).max()))
        a, e = a.reshape(-1, N, D)[:, -(N % 128):], e.reshape(-1, N, D)[:, -(N % 128):]  # the tile of the idle CTAs
        assert np.abs(a - e).max() <= 2e-2 + 4e-3 * np.abs(e).max(), name
    assert all(np.array_equal(x, y) for x, y in zip(got, again))
    assert ctx().device_status() == 0


@pytest.mark.parametrize("D,causal", [(64, True), (128, False)])
def test_backward_head_pairs(D, causal):
    """dQ with two heads to a CTA (4 * 148 pairs of query tiles) equals dQ of the same heads in a batch too small for that."""
    B, Hq, Hkv, N = 13, 32, 16, 260
    q, k, v, do = (torch.randn(B, h, N, D, generator=torch.Generator().manual_seed(h + i)).bfloat16().float().numpy()
                   for i, h in enumerate((Hq, Hkv, Hkv, Hq)))
    fo, fl = run_forward("grouped", fa.F32, fa.shape(B, Hq, Hkv, N, N, D), fa.config(causal), q.reshape(-1), k.reshape(-1), v.reshape(-1))
    fo = bf16_round(fo).reshape(B, Hq, N, D)
    flat = [x.reshape(-1) for x in (q, k, v, do, fo, fl)]
    dq, _, _ = run_backward(fa.BF16, B, Hq, Hkv, N, D, causal, None, *flat)
    dq = dq.reshape(B, Hq, N, D)
    fl = fl.reshape(B, Hq, N)
    for b in (0, B - 1):
        one, _, _ = run_backward(fa.BF16, 1, Hq, Hkv, N, D, causal, None, *(x[b].reshape(-1) for x in (q, k, v, do, fo, fl)))
        assert np.array_equal(dq[b].reshape(-1), one)


@pytest.mark.parametrize("S", [64, 65])
@pytest.mark.parametrize("dtype", [fa.BF16, fa.F16])
def test_padded_batches_around_the_lengths_that_travel_with_the_launch(S, dtype):
    """64 sequences' lengths and offsets are kernel arguments, 65 are copied to the workspace, where a decode plan that was
    uploaded before them must not be taken for granted.  Against the f32 kernel on the same rounded inputs."""
    Hq, Hkv, N, D, c = 4, 2, 70, 64, ctx()
    td = fa.torch_dtype(dtype)
    q, k, v = (torch.as_tensor(randn(S * N * h * D, 60 + i)).to(td).float().numpy() for i, h in enumerate((Hq, Hkv, Hkv)))
    rng = np.random.default_rng(S)
    lens = rng.integers(1, N + 1, S)
    lens[0], lens[-1] = N, 33
    seqs = [fa.VarlenSequence(int(n), int(n), 0, int(rng.integers(0, 3000))) for n in lens]
    cache = fa.CudaPagedKvCache(c, fa.BF16, 32, 160, Hkv, D)
    kv = torch.randn(2, 5000 * Hkv * D, generator=torch.Generator().manual_seed(S)).bfloat16().cuda()
    cache.record_append(kv[0], kv[1], 5000)
    dq, decoded = dev(randn(Hq * D, 70), torch.bfloat16), []

    def decode():
        out = c.create_decode_output_buffer(fa.BF16, 1, Hq, D)
        before = c.launch_count()
        c.decode_paged(fa.BF16, cache.table(), Hq, Hkv, D, fa.config(True), 5e5, 4999, dq, cache.k_buffer(), cache.v_buffer(), out)
        assert c.launch_count() - before == 2  # spans, whose plan lies in the workspace, and a merge
        decoded.append(out)

    shp, rot = fa.shape(S, Hq, Hkv, N, N, D), fa.rotary(5e5, 0)
    decode()
    o, l = run_forward("projection_rope_varlen", dtype, shp, fa.config(True), q, k, v, rot=rot, sequences=seqs)
    decode()
    assert torch.equal(*decoded)
    eo, el = run_forward("projection_rope_varlen", fa.F32, shp, fa.config(True), q, k, v, rot=rot, sequences=seqs)
    o, l, eo, el = o.reshape(S, N, Hq * D), l.reshape(S, Hq, N), eo.reshape(S, N, Hq * D), el.reshape(S, Hq, N)
    for b, n in enumerate(lens):
        assert np.abs(o[b, :n] - eo[b, :n]).max() <= 2e-2, b
        assert np.abs(l[b, :, :n] - el[b, :, :n]).max() <= 2e-3, b
        assert np.all(o[b, n:] == 0.0) and np.all(np.isneginf(l[b, :, n:])), b
    assert c.device_status() == 0


def test_exponent_of_head_dim_64_keeps_nan_and_zero():
    """A NaN query row stays NaN in O and LSE and alone; scores far below the row's maximum give exactly nothing."""
    B, H, N, D = 1, 2, 300, 64
    q, k, v = randn(B * H * N * D, 5), randn(B * H * N * D, 6), randn(B * H * N * D, 7)
    q.reshape(H, N, D)[1, 131] = np.nan
    k.reshape(H, N, D)[0, 7] = 60.0 * np.sign(q.reshape(H, N, D)[0, 9])  # one key far above all others for row 9
    q.reshape(H, N, D)[0, 9] = 60.0 * np.sign(q.reshape(H, N, D)[0, 9])
    o, l = run_forward("grouped", fa.BF16, fa.shape(B, H, H, N, N, D), fa.config(False), q, k, v)
    o, l = o.reshape(H, N, D), l.reshape(H, N)
    bad = np.zeros((H, N), bool)
    bad[1, 131] = True
    assert np.array_equal(np.isnan(l), bad) and np.array_equal(np.isnan(o).all(-1), bad) and np.array_equal(np.isnan(o).any(-1), bad)
    assert np.array_equal(o[0, 9], v.reshape(H, N, D)[0, 7])


@pytest.mark.parametrize("dtype", [fa.BF16, fa.F16])
def test_exponent_of_head_dim_64_is_accurate(dtype):
    """LSE of rows whose visible scores are 0 (key 0) and t (the 32 keys whose exponentials leave the special-function unit):
    log(1 + 32 e^t) shows an error of 2^t at full size."""
    H, N, D = 8, 128, 64
    td = fa.torch_dtype(dtype)
    a = torch.linspace(0, -64, H * N).to(td).double().reshape(H, N)  # t = a / 8 in the natural log domain: 2^0 to 2^-11.5
    a[0, :4] = torch.tensor([-704.0, -705.0, -2048.0, -30000.0]).to(td).double()  # below 2^-126.5
    q, k = torch.zeros(H, N, D), torch.zeros(H, N, D)
    q[:, :, 0], q[:, :, 1] = a.float(), 1.0
    k[:, 1:, 1] = -30000.0
    for j in range(N):
        if j % 8 >= 6:
            k[:, j, 0], k[:, j, 1] = 1.0, 0.0
    v = torch.ones(H, N, D)
    o, l = run_forward("grouped", dtype, fa.shape(1, H, H, N, N, D), fa.config(False), q.numpy(), k.numpy(), v.numpy())
    want = torch.log1p(32 * torch.exp(a / 8)).numpy()
    # 2^-22 for the exponentials, 2^-22 for the sum of 33 numbers, 2^-22 for t (the product of score, scale and log2 e, where the
    # sum depends on it), 2^-21 for log2 and the product with ln 2 at values up to 3.5
    assert np.abs(l.reshape(H, N) - want).max() <= 5 * 2.0 ** -22, np.abs(l.reshape(H, N) - want).max()
    assert np.all(l.reshape(H, N)[0, :4] == 0.0)
    assert np.all(np.abs(o - 1.0) <= 2.0 ** -8)


@pytest.mark.parametrize("H", [128, 130])
def test_alibi_slopes_of_many_heads(H):
    """Up to 128 slopes are kernel arguments, more are copied to the device."""
    N, D = 40, 64
    q, k, v = randn(N * H * D, 8), randn(N * H * D, 9), randn(N * H * D, 10)
    slopes = [float(2.0 ** (-8.0 * (h + 1) / H)) for h in range(H)]
    shp, c = fa.shape(1, H, H, N, N, D), ctx()
    out = c.create_output_buffer(fa.BF16, shp)
    c.forward_projection_rope_asymmetric_alibi(fa.BF16, shp, fa.config(True), fa.rotary(5e5, 0, 0), slopes, 0, 0,
                                               dev(q, torch.bfloat16), dev(k, torch.bfloat16), dev(v, torch.bfloat16), out)
    o, l = c.split_output(out, fa.BF16, shp, fa.PROJECTION)
    eo, el = ob.forward_reference_projection_grouped_rope_asymmetric_biased(q, k, v, ob._shape(1, H, H, N, N, D, 0), 5e5, 0, 0, causal=True,
                                                                            alibi=(slopes, 0, 0))
    assert np.abs(o.float().cpu().numpy().reshape(-1) - eo.reshape(-1)).max() <= 2e-2
    assert np.abs(l.cpu().numpy().reshape(-1) - el.reshape(-1)).max() <= 2e-3


def test_captured_calls_replay_to_the_same_bits():
    """Forward (rotation and attention), backward (three kernels) and decode (two) inside one CUDA graph: the launches that
    overlap in a stream keep their order in a graph."""
    B, Hq, Hkv, N, D = 2, 8, 2, 300, 128
    stream = torch.cuda.Stream()
    c = fa.Context(0, stream=stream)
    shp, cfg = fa.shape(B, Hq, Hkv, N, N, D), fa.config(True)
    q, k, v, do = (dev(randn(B * h * N * D, i), torch.bfloat16) for i, h in enumerate((Hq, Hkv, Hkv, Hq)))
    out = c.create_output_buffer(fa.BF16, shp)
    L = fa.backward_layout(fa.BF16, shp)
    packed, grads = c.empty_bytes(L.input_bytes), c.empty_bytes(L.output_bytes)
    for at, x in ((L.q_offset, q), (L.k_offset, k), (L.v_offset, v), (L.d_out_offset, do)):
        packed[at:at + 2 * x.numel()].view(torch.bfloat16).copy_(x.reshape(-1))
    cache = fa.CudaPagedKvCache(c, fa.BF16, 16, 50, Hkv, D)
    torch.cuda.synchronize()
    cache.record_append(k[:600 * Hkv * D], v[:600 * Hkv * D], 600)
    dec = c.create_decode_output_buffer(fa.BF16, 1, Hq, D)

    def calls():
        c.forward_grouped_rope(fa.BF16, shp, cfg, fa.rotary(5e5, 0, 0), q, k, v, out)
        c.forward_grouped(fa.BF16, shp, cfg, q, k, v, packed[L.out_offset:])
        c.backward_grouped(fa.BF16, shp, cfg, packed, grads)
        c.decode_paged(fa.BF16, cache.table(), Hq, Hkv, D, cfg, 5e5, 599, q[:Hq * D], cache.k_buffer(), cache.v_buffer(), dec)

    with torch.cuda.stream(stream):
        calls()  # tables and scratch
    torch.cuda.synchronize()
    want = [x.clone() for x in (out, grads, dec)]
    for x in (out, grads, dec):
        x.zero_()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        calls()
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip((out, grads, dec), want))
    assert c.device_status() == 0


# one forward kernel, rotation and forward, rotation, forward and merge of split parts; the tiled f32 kernel
@pytest.mark.parametrize("dtype,rope,H,N,D", [("BF16", False, 2, 100, 64), ("BF16", True, 4, 333, 128), ("F16", True, 2, 4096, 64),
                                              ("F32", True, 2, 200, 128)])
def test_calls_that_read_what_the_call_before_wrote(dtype, rope, H, N, D):
    """Calls overlap their launches with the end of the call before; what they read is complete all the same.  Each forward
    takes the output of the one before as Q, K and V."""
    c, code = ctx(), getattr(fa, dtype)
    td, shp = fa.torch_dtype(code), fa.shape(1, H, H, N, N, D)
    first = torch.randn(H * N * D, generator=torch.Generator().manual_seed(1)).to(td).cuda()
    outs = [c.create_output_buffer(code, shp) for _ in range(12)]

    def chain(between):
        x = first
        for out in outs:
            if rope:
                c.forward_grouped_rope(code, shp, fa.config(True), fa.rotary(5e5, 0, 0), x, x, x, out)
            else:
                c.forward_grouped(code, shp, fa.config(True), x, x, x, out)
            between()
            x = c.split_output(out, code, shp)[0].reshape(-1)
        torch.cuda.synchronize()
        return [out.clone() for out in outs]

    expected = chain(torch.cuda.synchronize)
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(chain(lambda: None), expected))
    assert c.device_status() == 0


@pytest.mark.parametrize("n", [40, 700, 9000])
def test_decode_steps_that_read_the_step_before(n):
    """The same for decode steps, in clusters and in spans with a merge: each takes the output of the one before as Q."""
    H, D, c = 8, 128, ctx()
    cache = fa.CudaResidentKvCache(c, fa.BF16, 1, H, n, D)
    g = torch.Generator().manual_seed(2)
    cache.record_append(*(torch.randn(n * H * D, generator=g).bfloat16().cuda() for _ in range(2)), n)
    first = torch.randn(H * D, generator=g).bfloat16().cuda()
    outs = [c.create_decode_output_buffer(fa.BF16, 1, H, D) for _ in range(30)]

    def chain(between):
        x = first
        for out in outs:
            c.decode_resident(fa.BF16, 1, H, H, D, n, n, fa.config(True), 5e5, n - 1, x, cache.k_buffer(), cache.v_buffer(), out)
            between()
            x = c.split_decode_output(out, fa.BF16, 1, H, D)[0].reshape(-1)
        torch.cuda.synchronize()
        return [out.clone() for out in outs]

    expected = chain(torch.cuda.synchronize)
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(chain(lambda: None), expected))
    assert c.device_status() == 0


def test_backward_that_reads_the_forward_before():
    """Training steps back to back: the gradients of each are those of its own forward."""
    B, Hq, Hkv, N, D, c = 2, 8, 2, 300, 64, ctx()
    shp, cfg = fa.shape(B, Hq, Hkv, N, N, D), fa.config(True)
    L = fa.backward_layout(fa.BF16, shp)
    packed, g = c.empty_bytes(L.input_bytes), torch.Generator().manual_seed(3)

    def view(at, count):
        return packed[at:at + 2 * count].view(torch.bfloat16)

    q, k, v, do = view(L.q_offset, L.q_elements), view(L.k_offset, L.kv_elements), view(L.v_offset, L.kv_elements), view(L.d_out_offset, L.q_elements)
    for x in (q, k, v, do):
        x.copy_(torch.randn(x.numel(), generator=g).bfloat16())
    start, grads = packed.clone(), [c.empty_bytes(L.output_bytes) for _ in range(10)]

    def steps(between):
        packed.copy_(start)
        for grad in grads:
            c.forward_grouped(fa.BF16, shp, cfg, q, k, v, packed[L.out_offset:])
            between()
            c.backward_grouped(fa.BF16, shp, cfg, packed, grad)
            between()
            c.forward_grouped(fa.BF16, shp, cfg, q, k, v, packed[L.out_offset:])  # O becomes the next step's Q
            between()
            q.copy_(view(L.out_offset, L.q_elements))
        torch.cuda.synchronize()
        return [x.clone() for x in grads]

    expected = steps(torch.cuda.synchronize)
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(steps(lambda: None), expected))
    assert c.device_status() == 0


# clusters of one tile per warp and of several, spans with a merge
@pytest.mark.parametrize("n", [40, 700, 9000])
@pytest.mark.parametrize("paged", [True, False])
def test_decode_of_tokens_that_the_call_before_appended(n, paged):
    """A serving loop appends and decodes: each step reads K and V that the call directly before it wrote, over and over at the
    same addresses and with other values each time."""
    Hq, Hkv, D, c, steps = 8, 8, 128, ctx(), 8
    cache = (fa.CudaPagedKvCache(c, fa.BF16, 16, (n + 15) // 16, Hkv, D) if paged else fa.CudaResidentKvCache(c, fa.BF16, 1, Hkv, n, D))
    g = torch.Generator(device="cuda").manual_seed(n)
    kv = [torch.randn(2, n * Hkv * D, generator=g, device="cuda").bfloat16() for _ in range(steps)]
    q = torch.randn(Hq * D, generator=g, device="cuda").bfloat16()
    outs = [c.create_decode_output_buffer(fa.BF16, 1, Hq, D) for _ in range(steps)]

    def loop(between):
        for (k, v), out in zip(kv, outs):
            cache.reset()
            cache.record_append(k, v, n)
            between()
            if paged:
                c.decode_paged(fa.BF16, cache.table(), Hq, Hkv, D, fa.config(True), 5e5, n - 1, q, cache.k_buffer(), cache.v_buffer(), out)
            else:
                c.decode_resident(fa.BF16, 1, Hq, Hkv, D, n, n, fa.config(True), 5e5, n - 1, q, cache.k_buffer(), cache.v_buffer(), out)
            between()
        torch.cuda.synchronize()
        return [out.clone() for out in outs]

    expected = loop(torch.cuda.synchronize)
    assert not torch.equal(expected[0], expected[1])
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(loop(lambda: None), expected))
    assert c.device_status() == 0


@pytest.mark.parametrize("n", [128, 700, 9000])
def test_decode_of_the_output_of_the_forward_before(n):
    """K and V of a decode are the output of the forward launched directly before it, whose last kernel lets its dependents
    start early."""
    H, D, c, steps = 8, 128, ctx(), 6
    shp = fa.shape(1, H, H, n, n, D)
    g = torch.Generator(device="cuda").manual_seed(n)
    x, q = (torch.randn(rows * H * D, generator=g, device="cuda").bfloat16() for rows in (n, 1))
    out = c.create_output_buffer(fa.BF16, shp)  # one buffer: the forward of a step overwrites what the decode before it read
    o = c.split_output(out, fa.BF16, shp, fa.PROJECTION)[0].reshape(-1)
    outs = [c.create_decode_output_buffer(fa.BF16, 1, H, D) for _ in range(steps)]

    def loop(between):
        for i, dec in enumerate(outs):
            c.forward_projection_rope_asymmetric(fa.BF16, shp, fa.config(i % 2 == 0), fa.rotary(5e5, 0, 0), x, x, x, out)
            between()
            c.decode_resident(fa.BF16, 1, H, H, D, n, n, fa.config(True), 5e5, n - 1, q, o, o, dec)
            between()
        torch.cuda.synchronize()
        return [dec.clone() for dec in outs]

    expected = loop(torch.cuda.synchronize)
    assert not torch.equal(expected[0], expected[1])
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(loop(lambda: None), expected))
    assert c.device_status() == 0


@pytest.mark.parametrize("dtype,rotate_k", [("BF16", True), ("BF16", False), ("F16", True), ("F32", True)])
def test_calls_that_fill_a_new_rotation_table(dtype, rotate_k):
    """Each call has other positions, so the (cos, sin) table that its first kernel reads was written directly before it."""
    H, N, D, c, code = 4, 200, 128, ctx(), getattr(fa, dtype)
    td, shp = fa.torch_dtype(code), fa.shape(1, H, H, N, N, D)
    g = torch.Generator().manual_seed(1)
    q, k, v = (torch.randn(N * H * D, generator=g).to(td).cuda() for _ in range(3))
    outs = [c.create_output_buffer(code, shp) for _ in range(10)]

    def loop(between):
        for i, out in enumerate(outs):
            c.forward_projection_rope_asymmetric(code, shp, fa.config(True), fa.rotary(5e5, 1000 * i + 7, 500 * i, rotate_k), q, k, v, out)
            between()
        torch.cuda.synchronize()
        return [out.clone() for out in outs]

    expected = loop(torch.cuda.synchronize)
    assert not torch.equal(expected[0], expected[1])
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(loop(lambda: None), expected))
    assert c.device_status() == 0


@pytest.mark.parametrize("kind", ["forward", "f32", "decode"])
def test_overlapped_calls_behind_another_stream(kind):
    """The context changes its stream, and a call's input comes from work of another stream that its own was made to wait for."""
    H, N, D, page = 4, 700, 128, 16
    code = fa.F32 if kind == "f32" else fa.BF16
    td, streams = fa.torch_dtype(code), [torch.cuda.Stream() for _ in range(2)]
    c, shp = fa.Context(0, stream=streams[0]), fa.shape(1, H, H, N, N, D)
    g = torch.Generator(device="cuda").manual_seed(1)
    a = torch.randn(2048, 2048, generator=g, device="cuda")
    x = torch.empty(N * H * D, dtype=td, device="cuda")
    outs = [c.create_decode_output_buffer(code, 1, H, D) if kind == "decode" else c.create_output_buffer(code, shp) for _ in range(10)]

    def call(out):
        if kind == "decode":
            c.decode_resident(code, 1, H, H, D, N, N, fa.config(True), 5e5, N - 1, x[:H * D], x, x, out)
        else:
            c.forward_grouped_rope(code, shp, fa.config(True), fa.rotary(5e5, 0), x, x, x, out)

    def loop(between):
        for i, out in enumerate(outs):
            mine, other = streams[i % 2], streams[1 - i % 2]
            mine.wait_stream(other)  # the scratch of the context is the call before's until then
            with torch.cuda.stream(other):
                other.wait_stream(mine)
                y = a
                for _ in range(4):
                    y = y @ a * 0.02
                x.copy_((y.reshape(-1)[:x.numel()] + i).to(td))
            mine.wait_stream(other)
            c.set_stream(mine)
            call(out)
            call(out)
            between()
        torch.cuda.synchronize()
        return [out.clone() for out in outs]

    expected = loop(torch.cuda.synchronize)
    assert not torch.equal(expected[0], expected[1])
    for _ in range(3):
        assert all(torch.equal(p, q) for p, q in zip(loop(lambda: None), expected))
    assert c.device_status() == 0
