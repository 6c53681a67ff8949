"""The register-tiled f32 forward (head_dim 64 / 128) at the edges of its 64-row blocks and 64-key tiles, with one CTA and
with a cluster of CTAs per block, against the CPU oracle (tolerances of the f32 RoPE tests)."""
import numpy as np
import pytest
import torch

from oracle import binding as ob
from tests.gpu_util import assert_close, ctx, dev, fa, ramp, run_forward

pytestmark = pytest.mark.gpu

ROPE_TOL = (1.5e-4, 1.0e-3)

SHAPES = [  # (B, Hq, Hkv, Nq, Nkv, D, causal, query offset)
    (1, 2, 1, 16, 16, 64, True, 0),
    (1, 2, 2, 63, 65, 128, False, 0),
    (1, 4, 2, 64, 64, 128, True, 0),
    (2, 4, 1, 65, 129, 64, True, 64),
    (1, 2, 1, 17, 700, 128, True, 683),
    (1, 8, 2, 130, 513, 64, False, 0),
    (3, 16, 16, 200, 200, 64, True, 0),
]


def case(B, Hq, Hkv, Nq, Nkv, D):
    return (ramp(B * Nq * Hq * D, 0.3, 0.071, 0.625, 0.3, 0.2), ramp(B * Nkv * Hkv * D, 0.9, 0.071, 0.625, 0.3, 0.2),
            ramp(B * Nkv * Hkv * D, 1.5, 0.071, 0.625, 0.3, 0.2))


@pytest.mark.parametrize("B,Hq,Hkv,Nq,Nkv,D,causal,coff", SHAPES)
def test_edges(B, Hq, Hkv, Nq, Nkv, D, causal, coff):
    q, k, v = case(B, Hq, Hkv, Nq, Nkv, D)
    shp = fa.shape(B, Hq, Hkv, Nq, Nkv, D, coff)
    o, l = run_forward("projection_rope_asymmetric", fa.F32, shp, fa.config(causal), q, k, v, rot=fa.rotary(5e5, coff, 0))
    eo, el = ob.forward_reference_projection_grouped_rope_asymmetric(q, k, v, ob._shape(B, Hq, Hkv, Nq, Nkv, D, coff), 5e5, coff, 0,
                                                                     causal)
    assert_close("O", o, eo, *ROPE_TOL)
    assert_close("LSE", l, el, *ROPE_TOL)


def test_a_call_under_capture_gives_the_same_bits():
    """The first call of a context under stream capture cannot allocate a rotation table: the kernel evaluates the angles."""
    B, Hq, Hkv, N, D = 1, 4, 2, 100, 128
    q, k, v = (dev(x) for x in case(B, Hq, Hkv, N, N, D))
    shp, cfg, rot = fa.shape(B, Hq, Hkv, N, N, D), fa.config(True), fa.rotary(5e5, 3, 3)
    want = ctx().create_output_buffer(fa.F32, shp)
    ctx().forward_projection_rope_asymmetric(fa.F32, shp, cfg, rot, q, k, v, want)
    stream = torch.cuda.Stream()
    c = fa.Context(0, stream=stream)
    got = c.create_output_buffer(fa.F32, shp)
    got.zero_()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        c.forward_projection_rope_asymmetric(fa.F32, shp, cfg, rot, q, k, v, got)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)


# (Hq, Hkv, Nq, Nkv, D, query offset), causal: one CTA per block, clusters, a diagonal that starts inside a tile
@pytest.mark.parametrize("Hq,Hkv,Nq,Nkv,D,coff", [(2, 1, 60, 60, 128, 0), (8, 2, 200, 200, 64, 0), (4, 4, 130, 330, 128, 200),
                                                  (2, 2, 100, 131, 64, 31)])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_non_finite_values_of_unseen_keys_stay_out(Hq, Hkv, Nq, Nkv, D, coff, bad):
    """A row is a function of the keys it sees: a non-finite V (and K) row changes no bit of the rows before it."""
    q, k, v = case(1, Hq, Hkv, Nq, Nkv, D)
    shp, cfg, rot = fa.shape(1, Hq, Hkv, Nq, Nkv, D, coff), fa.config(True), fa.rotary(5e5, coff, 0)
    o, l = (x.reshape(s) for x, s in zip(run_forward("projection_rope_asymmetric", fa.F32, shp, cfg, q, k, v, rot=rot),
                                         ((Nq, Hq, D), (Hq, Nq))))
    for key in (40, 63, 64, Nkv - 1):
        if key >= Nkv:
            continue
        first = max(0, key - coff)  # the first row that sees the key
        v2 = v.reshape(Nkv, Hkv, D).copy()
        v2[key] = bad
        o2, l2 = run_forward("projection_rope_asymmetric", fa.F32, shp, cfg, q, k, v2, rot=rot)
        o2, l2 = o2.reshape(Nq, Hq, D), l2.reshape(Hq, Nq)
        assert np.array_equal(o2[:first], o[:first]), (key, int(np.isnan(o2).any((1, 2)).argmax()))
        assert np.array_equal(l2, l)
        assert not np.isfinite(o2[first:]).any()
        k2 = k.reshape(Nkv, Hkv, D).copy()
        k2[key] = bad
        o2, l2 = run_forward("projection_rope_asymmetric", fa.F32, shp, cfg, q, k2, v, rot=rot)
        assert np.array_equal(o2.reshape(Nq, Hq, D)[:first], o[:first])
        assert np.array_equal(l2.reshape(Hq, Nq)[:, :first], l[:, :first])


def f32_rope_call(c, D, N, theta, pos):
    """One f32 RoPE forward of 4 / 2 heads with queries and keys from position `pos` on, into a buffer of its own."""
    q, k, v = (dev(x) for x in case(1, 4, 2, N, N, D))
    shp = fa.shape(1, 4, 2, N, N, D)
    out = c.create_output_buffer(fa.F32, shp)
    out.zero_()
    c.forward_grouped_rope(fa.F32, shp, fa.config(True), fa.rotary(theta, pos, pos), q, k, v, out)
    torch.cuda.synchronize()
    return out


def test_f32_calls_of_changing_positions_give_the_bits_of_a_fresh_context():
    """The table of one range serves the ranges inside it, another theta, head_dim or range replaces it; beyond its size the
    kernel evaluates the angles."""
    c = fa.Context(0)
    calls = [(128, 100, 5e5, 0), (128, 60, 5e5, 17), (128, 120, 5e5, 0), (128, 100, 5e5, 4000), (64, 100, 5e5, 4000),
             (64, 100, 1e4, 4000), (128, 100, 5e5, 0), (128, 100, 5e5, 1 << 20)]
    for i, (D, N, theta, pos) in enumerate(calls):
        assert torch.equal(f32_rope_call(c, D, N, theta, pos), f32_rope_call(fa.Context(0), D, N, theta, pos)), i
    D, Nq, Nkv = 128, 16, 33000  # more positions than the table holds, of which the mask leaves 1000
    q, k, v = (dev(x) for x in case(1, 2, 1, Nq, Nkv, D))
    rows = []
    for n in (1000, Nkv):
        shp = fa.shape(1, 2, 1, Nq, n, D, 984)
        out = c.create_output_buffer(fa.F32, shp)
        c.forward_projection_rope_asymmetric(fa.F32, shp, fa.config(True), fa.rotary(5e5, 984, 0), q, k[:n * D], v[:n * D], out)
        rows.append(out)
    torch.cuda.synchronize()
    assert torch.equal(*rows)


def test_a_captured_16_bit_call_replays_unchanged_after_f32_calls():
    """A captured RoPE call of the tensor-core kernel holds the address of a (cos, sin) table: f32 calls leave those alone."""
    B, Hq, Hkv, N, D = 1, 4, 2, 300, 128
    stream = torch.cuda.Stream()
    c = fa.Context(0, stream=stream)
    c.reserve_rope_tables(512, D)  # nothing below frees a table, whoever writes to it
    shp, cfg, rot = fa.shape(B, Hq, Hkv, N, N, D), fa.config(True), fa.rotary(5e5, 7, 7)
    q, k, v = (dev(x, torch.bfloat16) for x in case(B, Hq, Hkv, N, N, D))
    out = c.create_output_buffer(fa.BF16, shp)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        c.forward_grouped_rope(fa.BF16, shp, cfg, rot, q, k, v, out)
        torch.cuda.synchronize()
        want = out.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        c.forward_grouped_rope(fa.BF16, shp, cfg, rot, q, k, v, out)
    for pos in (100, 200):
        f32_rope_call(c, D, 250, 5e5, pos)
    out.zero_()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)


def test_f32_calls_do_not_trust_a_table_that_a_graph_fills():
    """A 16-bit call captured before its (cos, sin) table exists fills it in each replay, and not before the first."""
    stream = torch.cuda.Stream()
    c = fa.Context(0, stream=stream)
    N, D, pos = 200, 128, 50
    c.reserve_rope_tables(256, D)
    shp = fa.shape(1, 4, 2, N, N, D)
    q, k, v = (dev(x, torch.bfloat16) for x in case(1, 4, 2, N, N, D))
    out = c.create_output_buffer(fa.BF16, shp)
    c.prepare_forward(fa.BF16, fa.HEAD_MAJOR, shp, fa.config(True), fa.rotary(5e5, pos, pos), q, k, v, out)  # the scratch
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        c.forward_grouped_rope(fa.BF16, shp, fa.config(True), fa.rotary(5e5, pos, pos), q, k, v, out)
    want = f32_rope_call(fa.Context(0), D, N, 5e5, pos)
    assert torch.equal(f32_rope_call(c, D, N, 5e5, pos), want)
    graph.replay()
    assert torch.equal(f32_rope_call(c, D, N, 5e5, pos), want)


def test_an_f32_prepared_pass_allocates_nothing():
    """flat_forward_encode_prepared: no allocation, without any reservation before it.  16 rows against 32000 keys, whose
    (cos, sin) take 16 MB of device memory."""
    c = fa.Context(0)
    Hq, Hkv, Nq, Nkv, D = 2, 1, 16, 32000, 128
    q, k, v = (dev(x) for x in case(1, Hq, Hkv, Nq, Nkv, D))
    shp, cfg, rot = fa.shape(1, Hq, Hkv, Nq, Nkv, D, Nkv - Nq), fa.config(True), fa.rotary(5e5, Nkv - Nq, 0)
    out, want = c.create_output_buffer(fa.F32, shp), c.create_output_buffer(fa.F32, shp)
    prepared = c.prepare_forward(fa.F32, fa.PROJECTION, shp, cfg, rot, q, k, v, out)
    torch.cuda.synchronize()
    free, workspace = torch.cuda.mem_get_info()[0], c.workspace_bytes()
    prepared.encode()
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free and c.workspace_bytes() == workspace
    fa.Context(0).forward_projection_rope_asymmetric(fa.F32, shp, cfg, rot, q, k, v, want)
    torch.cuda.synchronize()
    assert torch.equal(out, want)
