"""Tile edges of the grouped contraction kernel: token counts around its tile widths, weight rows that fill no whole
tile, blocks with holes.  The tensor-core path against the CUDA-core kernels on the same quantised inputs.

Tolerance, as max|a - b| / max|b|: both sides round each output to bf16 (half a step each, together 2^-8), and where an
intermediate lies on a rounding tie of its e4m3 code the two summation orders may take different sides, which moves an
output by 2^-4 of one of its I >= 32 terms; 1e-2 covers both with a factor of two."""

import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 1e-2


def _blocks(counts, B, holes):
    """token_position_to_id / block_to_expert for ``counts[e]`` tokens of expert e, ids in order of position; with
    ``holes`` the first block of an expert that has several is left half empty."""
    tpi, b2e, t = [], [], 0
    for e, n in enumerate(counts):
        left = n
        while left > 0:
            take = min(left, B // 2 - 3 if holes and left == n and n > B else B)
            tpi += list(range(t, t + take)) + [-1] * (B - take)
            b2e.append(e)
            t, left = t + take, left - take
    i32 = dict(dtype=torch.int32, device="cuda")
    return torch.tensor(tpi, **i32), torch.tensor(b2e, **i32), t


@pytest.mark.parametrize("variant", ["single", "pair"])
@pytest.mark.parametrize("counts,B,H,I,holes", [
    ([1, 15, 16, 17, 0, 31, 33], 128, 256, 32, False),
    ([127, 128, 129, 255], 128, 128, 96, False),
    ([223, 224, 225, 1], 256, 160, 416, False),
    ([256, 257, 448, 449, 513], 256, 128, 160, False),
    ([700, 3, 300], 128, 256, 64, True),
])
def test_tile_edges(variant, counts, B, H, I, holes):
    import nki_library_b200 as m
    from nki_library_b200 import _lib
    from nki_library_b200.layer import random_expert_weights
    tpi, b2e, T = _blocks(counts, B, holes)
    E = len(counts)
    g = torch.Generator(device="cuda").manual_seed(T + I)
    w = random_expert_weights(E, H, I, "cuda", seed=I)
    w.bias_gu = torch.randn((E, 2 * I), device="cuda", generator=g) * 0.5
    w.bias_d = torch.randn((E, H), device="cuda", generator=g) * 0.5
    x = torch.randn((T, H), device="cuda", generator=g).to(torch.bfloat16)
    aff = torch.rand((T, E), device="cuda", generator=g)

    def run(impl):
        return m.moe_cte(x, aff.view(-1, 1), w, None, tpi, b2e, B, m.MoECTESpec(m.MoECTEImplementation.shard_on_block_mx),
                         skip_dma=m.SkipMode(True, False), _impl=impl, _check_status=True).float()

    ref = run(_lib.IMPL_SIMT)
    got = run(_lib.GEMM_NO_PAIR if variant == "single" else _lib.GEMM_FORCE_PAIR)
    assert float((got - ref).abs().max() / ref.abs().max()) <= TOL


@pytest.mark.parametrize("variant", ["single", "pair"])
@pytest.mark.parametrize("weights", ["e4m3", "e2m1", "bf16"])
def test_many_tiles_per_cta(variant, weights):
    """Every CTA walks several tiles of both contractions: token tiles wider than one accumulator between narrower ones, rows
    of several experts through the same output buffers, a last round that single CTAs cut.  All outputs are compared."""
    import nki_library_b200 as m
    from nki_library_b200 import _lib
    from nki_library_b200.layer import random_expert_weights
    from nki_library_b200.weights import prepare_dense
    counts, B, H, I = [256, 225, 224, 31, 480, 1, 449, 700, 0, 130, 65, 288] * 2, 256, 2048, 1024
    tpi, b2e, T = _blocks(counts, B, False)
    E = len(counts)
    g = torch.Generator(device="cuda").manual_seed(8)
    if weights == "bf16":
        w = prepare_dense(*((torch.randn(s, device="cuda", generator=g) * 0.02).to(torch.bfloat16)
                            for s in ((E, H, 2, I), (E, I, H))))
    else:
        w = random_expert_weights(E, H, I, "cuda", seed=6, w_format=5 if weights == "e2m1" else 0)
    w.bias_gu = torch.randn((E, 2 * I), device="cuda", generator=g) * 0.5
    w.bias_d = torch.randn((E, H), device="cuda", generator=g) * 0.1
    x = torch.randn((T, H), device="cuda", generator=g).to(torch.bfloat16)
    aff = torch.rand((T, E), device="cuda", generator=g) + 0.5
    spec = m.MoECTESpec(m.MoECTEImplementation.shard_on_block if weights == "bf16" else
                        m.MoECTEImplementation.shard_on_block_mx)

    def run(impl):
        return m.moe_cte(x, aff.view(-1, 1), w, None, tpi, b2e, B, spec, skip_dma=m.SkipMode(True, False), _impl=impl,
                         _check_status=True)

    ref = run(_lib.IMPL_SIMT).float()
    impl = _lib.GEMM_NO_PAIR if variant == "single" else _lib.GEMM_FORCE_PAIR
    got = run(impl)
    assert float((got.float() - ref).abs().max() / ref.abs().max()) <= TOL
    assert torch.equal(run(impl), got)


def test_clock_probe_times_its_own_launch():
    """A probed contraction does not start inside the launch in front, whose rest it would count.  In front stands a long
    RMSNorm that leaves most SMs idle and lets chained launches in at once."""
    from nki_library_b200 import _lib, pipeline
    from nki_library_b200.layer import random_expert_weights
    H, I = 128, 128
    w = random_expert_weights(1, H, I, "cuda", seed=1)
    ws = pipeline.BlockWorkspace(128, H, I, "cuda")
    ws.xq.zero_()
    ws.tile_flags.fill_(128)
    b2e = torch.zeros(1, dtype=torch.int32, device="cuda")
    probe = torch.zeros(2, dtype=torch.int64, device="cuda")
    rows, cols = 32, 1 << 24
    x = torch.zeros((rows, cols), dtype=torch.bfloat16, device="cuda")
    out = torch.empty_like(x)
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    nan = float("nan")
    for _ in range(2):
        torch.cuda.synchronize()
        ev[0].record()
        _lib.call("b200moe_rmsnorm", _lib.ptr(x), None, None, _lib.F32, rows, cols, 0, 1e-6, _lib.ptr(out), None,
                  _lib.stream_ptr())
        _lib.call("b200moe_grouped_gemm1_swiglu", _lib.ptr(ws.xq), _lib.ptr(ws.x_sf), _lib.ptr(w.w1), _lib.ptr(w.w1_sf),
                  w.w_format, None, _lib.ptr(b2e), None, _lib.ptr(ws.tile_flags), 1, 128, 1, H, I, 0, nan, nan, nan, nan,
                  _lib.ptr(ws.mq), _lib.ptr(ws.m_sf), _lib.ptr(ws.status) + 4, _lib.GEMM_CHAINED, _lib.ptr(probe),
                  _lib.stream_ptr())
        ev[1].record()
    torch.cuda.synchronize()
    assert ws.status.tolist()[1] == 0
    assert 0 < int(probe[1]) < 0.2e6 * ev[0].elapsed_time(ev[1])  # nanoseconds against a fifth of milliseconds


@pytest.mark.parametrize("variant", ["single", "pair"])
@pytest.mark.parametrize("act", [0, 3])
def test_gate_up_of_extreme_products(variant, act):
    """MX blocks of gate/up products that are zero, subnormal, huge, infinite or NaN.  The weights are zero, so the biases
    are the gates and ups; scales and codes against the CUDA-core kernel (values are no rounding ties of either)."""
    from nki_library_b200 import _lib, pipeline
    from nki_library_b200.weights import ExpertWeights
    E, H, I, B = 7, 128, 128, 256
    f = dict(dtype=torch.float32, device="cuda")
    j = torch.arange(I, **f)
    gate, up = (j % 13 - 6.1).repeat(E, 1), (j % 7 - 2.9).repeat(E, 1)
    gate[1, 37] = float("nan")
    up[2, 5] = float("inf")
    gate[2, 70] = float("-inf")
    gate[3] = 0.0
    gate[4] = 3e-39
    gate[5], up[5] = 1.5e30, 2.5e8
    up[6, 64:96] = 1e-38
    bias = torch.stack([gate, up], 1).view(E, 2, I // 32, 32).transpose(1, 2).reshape(E, 2 * I).contiguous()
    lib = _lib.load_library()
    zeros = [torch.zeros(n, dtype=torch.uint8, device="cuda") for n in
             (E * 2 * I * H, E * lib.b200moe_sf_bytes(2 * I, H), E * H * I, E * lib.b200moe_sf_bytes(H, I))]
    w = ExpertWeights(E, H, I, *zeros, bias, None, False)
    b2e = torch.arange(E, dtype=torch.int32, device="cuda")
    nan = float("nan")

    def run(impl):
        ws = pipeline.BlockWorkspace(E * B, H, I, "cuda")
        for t in (ws.xq, ws.mq):
            t.zero_()
        ws.tile_flags.fill_(128)
        _lib.call("b200moe_grouped_gemm1_swiglu", _lib.ptr(ws.xq), _lib.ptr(ws.x_sf), _lib.ptr(w.w1), _lib.ptr(w.w1_sf),
                  w.w_format, _lib.ptr(w.bias_gu), _lib.ptr(b2e), None, _lib.ptr(ws.tile_flags), E, B, E, H, I, act, nan, nan,
                  nan, nan, _lib.ptr(ws.mq), _lib.ptr(ws.m_sf), _lib.ptr(ws.status) + 4, impl, None, _lib.stream_ptr())
        assert ws.status.tolist()[1] == 0
        code = ws.mq & 0x7F
        return torch.where(code == 0x7F, code, ws.mq), ws.m_sf  # a NaN's sign says nothing

    ref = run(_lib.IMPL_SIMT)
    got = run(_lib.GEMM_NO_PAIR if variant == "single" else _lib.GEMM_FORCE_PAIR)
    assert torch.equal(got[1], ref[1])
    assert torch.equal(got[0], ref[0])
