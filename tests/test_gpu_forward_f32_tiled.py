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
