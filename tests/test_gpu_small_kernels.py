"""The bookkeeping and row kernels around the contractions at the edges of their loops: position lists longer than one
round, columns past a whole number of vectors, more chunks than one thread scans.  Integer results and copies are
compared exactly; the RMSNorm against fp64 torch within one bf16 rounding (2^-8 of the value) and the combine with the
fp32 sum in the same order."""

import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu


def _lib():
    from nki_library_b200 import _lib
    return _lib


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _positions(T, K, n_pos, share, seed):
    """[T, K] table of distinct positions, a share of the entries empty, some of those out of range."""
    g = _gen(seed)
    table = torch.randperm(n_pos, device="cuda", generator=g)[:T * K].reshape(T, K).to(torch.int32)
    drop = torch.rand((T, K), device="cuda", generator=g) >= share
    return torch.where(drop, torch.where(torch.arange(K, device="cuda") % 2 == 0, -1, n_pos + 5).to(torch.int32), table)


@pytest.mark.parametrize("T,H,K,share", [(3, 512, 1, 1.0), (9, 1024, 8, 1.0), (17, 1152, 33, 0.3), (5, 2176, 129, 0.1),
                                         (2, 3072, 300, 0.5)])
@pytest.mark.parametrize("packed", [0, 1])
def test_scatter_quantize_long_lists(T, H, K, share, packed):
    L = _lib()
    H = (H + 511) // 512 * 512 if packed else H
    n_pos = (T * K + 127) // 128 * 128
    table = _positions(T, K, n_pos, share, H + K)
    x = torch.randn((T, H), device="cuda", generator=_gen(1)).to(torch.bfloat16)
    nsf = L.load_library().b200moe_sf_bytes(n_pos, H)

    def buffers():
        return (torch.zeros((n_pos, H), dtype=torch.uint8, device="cuda"), torch.zeros(nsf, dtype=torch.uint8, device="cuda"),
                torch.zeros((n_pos // 128,), dtype=torch.int32, device="cuda"))

    got = buffers()
    L.call("b200moe_scatter_quantize_mxfp8", L.ptr(x), T, H, L.ptr(table), K, n_pos, packed, *map(L.ptr, got), L.stream_ptr())
    # the position-major kernel on the forward map of the same table
    tpi = torch.full((n_pos,), -1, dtype=torch.int32, device="cuda")
    ok = (table >= 0) & (table < n_pos)
    tpi[table[ok].long()] = torch.arange(T, dtype=torch.int32, device="cuda")[:, None].expand(T, K)[ok]
    ref = buffers()
    L.call("b200moe_gather_quantize_mxfp8", L.ptr(x), T, H, L.ptr(tpi), n_pos, packed, *map(L.ptr, ref), L.stream_ptr())
    held = tpi >= 0
    assert torch.equal(got[0][held], ref[0][held]) and torch.equal(got[2], ref[2])
    pos = torch.arange(n_pos, device="cuda")
    kb = torch.arange(H // 32, device="cuda")
    at = (((pos >> 7)[:, None] * ((H + 127) // 128) + (kb >> 2)[None]) * 512 + (pos & 31)[:, None] * 16 +
          (((pos >> 5) & 3) * 4)[:, None] + (kb & 3)[None])
    assert torch.equal(got[1][at][held], ref[1][at][held])


@pytest.mark.parametrize("T,H,K", [(1, 8, 1), (7, 1032, 3), (11, 4104, 130)])
@pytest.mark.parametrize("scaled", [False, True])
def test_scatter_rows(T, H, K, scaled):
    L = _lib()
    B, E = 128, 5
    n_pos = (T * K + B - 1) // B * B
    table = _positions(T, K, n_pos, 0.6, H)
    x = torch.randn((T, H), device="cuda", generator=_gen(2)).to(torch.bfloat16)
    b2e = torch.randint(0, E, (n_pos // B,), dtype=torch.int32, device="cuda", generator=_gen(3))
    aff = torch.rand((T, E), device="cuda", generator=_gen(4))
    out = torch.zeros((n_pos, H), dtype=torch.bfloat16, device="cuda")
    flags = torch.empty((n_pos // 128,), dtype=torch.int32, device="cuda")
    L.call("b200moe_scatter_rows_bf16", L.ptr(x), T, H, L.ptr(table), K, n_pos, L.ptr(b2e), B, E,
           L.ptr(aff) if scaled else None, L.F32, L.ptr(out), L.ptr(flags), L.stream_ptr())
    ref = torch.zeros_like(out)
    want = torch.zeros_like(flags)
    for t in range(T):
        for p in table[t].tolist():
            if 0 <= p < n_pos:
                a = aff[t, int(b2e[p // B])].to(torch.bfloat16).float() if scaled else 1.0
                ref[p] = (x[t].float() * a).to(torch.bfloat16)
                want[p >> 7] = max(int(want[p >> 7]), (p & 127) + 1)
    assert torch.equal(out, ref) and torch.equal(flags, want)


@pytest.mark.parametrize("T,H,offset", [(1, 8, 0), (5, 250, 0), (3, 1001, 0), (4, 4096, 0), (2, 9000, 0), (3, 512, 1)])
@pytest.mark.parametrize("residual", [False, True])
def test_rmsnorm_odd_rows(T, H, offset, residual):
    """Row lengths that are no multiple of a vector or of the CTA, and rows that start off a 16-byte boundary."""
    L = _lib()
    x = torch.randn((T * H + offset,), device="cuda", generator=_gen(5)).to(torch.bfloat16)[offset:].view(T, H)
    r = torch.randn((T, H), device="cuda", generator=_gen(6)).to(torch.bfloat16) if residual else None
    gamma = torch.rand((H,), device="cuda", generator=_gen(7)) + 0.5
    out, res = torch.empty((T, H), dtype=torch.bfloat16, device="cuda"), torch.empty((T, H), dtype=torch.bfloat16, device="cuda")
    L.call("b200moe_rmsnorm", L.ptr(x), L.ptr(r), L.ptr(gamma), L.F32, T, H, 0, 1e-6, L.ptr(out),
           L.ptr(res) if residual else None, L.stream_ptr())
    v = (x.float() + r.float()).to(torch.bfloat16) if residual else x
    if residual:
        assert torch.equal(res, v)
    ref = v.double() / torch.sqrt(v.double().pow(2).mean(1, keepdim=True) + 1e-6) * gamma.double()
    assert bool(((out.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-30).all())


@pytest.mark.parametrize("T,n_cand,H", [(1, 1, 8), (3, 7, 1032), (2, 9, 3072), (5, 130, 2056), (1200, 17, 256), (1300, 2, 1032)])
def test_combine_lists(T, n_cand, H):
    L = _lib()
    rows = T * n_cand
    y = torch.randn((rows, H), device="cuda", generator=_gen(8)).to(torch.bfloat16)
    table = _positions(T, n_cand, rows, 0.7, T)
    table = torch.where(table >= rows, -1, table)
    out = torch.empty((T, H), dtype=torch.bfloat16, device="cuda")
    L.call("b200moe_combine", L.ptr(y), L.ptr(table), T, n_cand, H, L.ptr(out), L.stream_ptr())
    ref = torch.zeros((T, H), dtype=torch.float32, device="cuda")
    for c in range(n_cand):
        p = table[:, c]
        ref = ref + torch.where((p >= 0)[:, None], y[p.clamp(min=0).long()].float(), 0.0)
    assert torch.equal(out, ref.to(torch.bfloat16))


@pytest.mark.parametrize("T,E,K,B", [(1, 1, 1, 128), (256, 33, 3, 128), (257, 4, 2, 128), (2305, 17, 5, 256),
                                     (4500, 513, 8, 128), (9000, 128, 8, 128), (700, 1000, 4, 128)])
def test_group_tokens_scan(T, E, K, B):
    """Chunks of 256 tokens are scanned by several threads per column when the columns leave room for that."""
    import nki_library_b200 as m
    idx = torch.rand((T, E), device="cuda", generator=_gen(T)).topk(K, dim=1).indices.to(torch.int32)
    N = m.get_n_blocks(T, K, E, B)
    g = m.moe_group_tokens(idx, E, B, N, top_k=K, check=True)
    tpi, b2e, pos, counts = [], [], torch.full((T, E), -1, dtype=torch.int64), []
    sel = torch.zeros((T, E), dtype=torch.bool)
    sel.scatter_(1, idx.cpu().long(), True)
    for e in range(E):
        ids = sel[:, e].nonzero().flatten()
        blocks = (len(ids) + B - 1) // B
        pos[ids, e] = len(tpi) + torch.arange(len(ids))
        tpi += ids.tolist() + [-1] * (blocks * B - len(ids))
        b2e += [e] * blocks
        counts.append(len(ids))
    used = len(b2e)
    tpi += [-1] * ((N - used) * B)
    b2e += [E - 1] * (N - used)
    assert g["token_position_to_id"].tolist() == tpi and g["block_to_expert"].tolist() == b2e
    assert g["counts"].tolist() == counts and g["conditions"].tolist() == [1] * used + [0] * (N - used + 2)
    assert torch.equal(g["inverse_map"].cpu().long(), pos.gather(1, idx.cpu().long()))
    # too few blocks are reported
    if used > 1:
        assert int(m.moe_group_tokens(idx, E, B, used - 1, top_k=K)["status"]) == 1


@pytest.mark.parametrize("T,E_L,E,rank_dtype", [(1, 1, 1, torch.int32), (129, 16, 128, torch.int32), (37, 3, 10, torch.int64),
                                                (128, 128, 128, torch.uint8)])
@pytest.mark.parametrize("masked", [False, True])
def test_all_expert_setup(T, E_L, E, rank_dtype, masked):
    mod = importlib.import_module("nki_library_b200.core.moe.moe_tkg.moe_tkg")
    r = E // E_L - 1
    K = min(4, E)
    aff = torch.rand((T, E), device="cuda", generator=_gen(11)).to(torch.bfloat16 if E == 10 else torch.float32)
    idx = torch.rand((T, E), device="cuda", generator=_gen(12)).topk(K, dim=1).indices
    rank = torch.tensor([[r]], dtype=rank_dtype, device="cuda")
    got = mod.local_affinities(aff, E_L, T, rank, idx.to(torch.int32) if masked else None)
    sel = torch.zeros((T, E), device="cuda").scatter_(1, idx, 1.0) if masked else 1.0
    assert torch.equal(got, (aff.float() * sel)[:, r * E_L:(r + 1) * E_L])
    tpi, b2e, table = mod.all_expert_layout(T, E_L, aff.device)
    pad = (T + 127) // 128 * 128
    ids = torch.full((pad,), -1, dtype=torch.int32, device="cuda")
    ids[:T] = torch.arange(T, device="cuda")
    assert torch.equal(tpi, ids.repeat(E_L))
    assert b2e.tolist() == [e for e in range(E_L) for _ in range(pad // 128)]
    assert torch.equal(table, (torch.arange(E_L, device="cuda")[None] * pad + torch.arange(T, device="cuda")[:, None]).int())


@pytest.mark.parametrize("E", [1, 3, 4, 12, 65, 250, 511])
def test_router_narrow_and_odd_widths(E):
    """Router weight rows that are no whole number of 16-byte pieces; ids exact, logits within the fp32 sum's error."""
    import nki_library_b200 as m
    T, H = 37, 640
    x = torch.randn((T, H), device="cuda", generator=_gen(9)).to(torch.bfloat16)
    w = (torch.randn((H, E), device="cuda", generator=_gen(10)) * 0.1).to(torch.bfloat16)
    k = min(E, 4)
    logits, aff = torch.empty((T, E), device="cuda"), torch.empty((T, E), device="cuda")
    idx = torch.empty((T, k), dtype=torch.int32, device="cuda")
    m.router_topk(x, w, None, logits, aff, idx, m.RouterActFnType.SOFTMAX, k, 1, 0, norm_topk_prob=True)
    ref = x.double() @ w.double()
    # H products added in fp32: at most H * 2^-24 of the sum of magnitudes
    assert bool(((logits.double() - ref).abs() <= H * 2.0 ** -24 * (x.double().abs() @ w.double().abs())).all())
    assert torch.equal(idx.long(), logits.topk(k, dim=1).indices)
    p = torch.softmax(logits, 1).gather(1, idx.long())
    want = torch.zeros_like(aff).scatter_(1, idx.long(), p / p.sum(1, keepdim=True))
    assert bool(((aff - want).abs() <= 1e-5 * want + 1e-12).all())


@pytest.mark.parametrize("T,E,K,B", [(3, 128, 8, 128), (256, 5, 2, 256), (3000, 40, 4, 128), (3000, 3, 1, 512)])
def test_tile_flags_from_bookkeeping(T, E, K, B):
    """The occupied rows per 128 positions, from the grouping and from the position table, are what the quantiser's
    stores say."""
    import nki_library_b200 as m
    L = _lib()
    idx = torch.rand((T, E), device="cuda", generator=_gen(T + E)).topk(K, dim=1).indices.to(torch.int32)
    N = m.get_n_blocks(T, K, E, B)
    flags = torch.full((N * B // 128,), 77, dtype=torch.int32, device="cuda")
    g = m.moe_group_tokens(idx, E, B, N, top_k=K, _tile_flags=flags)
    rows = torch.arange(128, device="cuda") + 1
    want = ((g["token_position_to_id"].view(-1, 128) >= 0) * rows).amax(1).int()
    assert torch.equal(flags, want)
    table = torch.empty((T, E), dtype=torch.int32, device="cuda")
    flags.fill_(77)
    L.call("b200moe_build_position_table_tiles", L.ptr(g["token_position_to_id"]), L.ptr(g["block_to_expert"]),
           L.ptr(g["conditions"]), N, B, T, E, L.ptr(table), L.ptr(flags), L.stream_ptr())
    assert torch.equal(flags, want)
    assert torch.equal(table.gather(1, idx.long()), g["inverse_map"])


@pytest.mark.parametrize("act", ["SOFTMAX", "SIGMOID"])
@pytest.mark.parametrize("mode", ["norm", "pre", "post"])
@pytest.mark.parametrize("E,k", [(8, 8), (33, 3), (128, 8), (512, 1)])
def test_router_winner_lanes(act, mode, E, k):
    """Winners are activated and written by their own lanes: every pipeline, ties, -0 and -inf logits (from the bias)."""
    import nki_library_b200 as m
    T, H = 19, 256
    x = torch.randn((T, H), device="cuda", generator=_gen(13)).to(torch.bfloat16)
    x[0] = 0  # all logits are the bias: ties
    w = (torch.randn((H, E), device="cuda", generator=_gen(14)) * 0.1).to(torch.bfloat16)
    bias = torch.zeros((E,), device="cuda", dtype=torch.bfloat16)
    bias[1::3] = -0.0
    bias[E - 1] = float("-inf")
    logits, aff = torch.empty((T, E), device="cuda"), torch.full((T, E), 9.0, device="cuda")
    idx = torch.empty((T, k), dtype=torch.int32, device="cuda")
    m.router_topk(x, w, bias, logits, aff, idx, m.RouterActFnType[act], k, 1, 0, router_pre_norm=mode != "post",
                  norm_topk_prob=mode == "norm", use_indirect_dma_scatter=True)
    order = torch.sort(logits + 0.0, dim=1, descending=True, stable=True).indices[:, :k]
    assert torch.equal(idx.long(), order)
    top = logits.gather(1, order).double()
    if act == "SIGMOID":
        val, full = torch.sigmoid(top), torch.sigmoid(logits.double())
    else:
        full = torch.softmax(logits.double(), 1)
        val = full.gather(1, order) if mode != "post" else torch.softmax(top, 1)
    if mode == "norm":
        val = val / val.sum(1, keepdim=True)
    want = full if mode == "pre" else torch.zeros_like(full).scatter_(1, order, val)
    # a handful of fp32 operations per value, exponents of up to ~10: 1e-5 relative
    assert bool(((aff.double() - want).abs() <= 1e-5 * want + 1e-12).all())


@pytest.mark.parametrize("T", [1, 16, 64])
def test_router_sum_order(T):
    """A split of the hidden axis holds at least 256 columns; inside one the products are added in fp32, the splits' sums in
    order.  2^24 in the first split swallows a 1 that is added alone, not a 2: each later split holds two ones, 128 columns
    apart."""
    import nki_library_b200 as m
    H, E = 1024, 8
    x, w = torch.zeros((T, H), device="cuda"), torch.zeros((H, E), device="cuda")
    x[:, 0], w[0] = 4096.0, 4096.0
    for s in (256, 512, 768):
        x[:, s], x[:, s + 128], w[s], w[s + 128] = 1.0, 1.0, 1.0, 1.0
    logits, aff = torch.empty((T, E), device="cuda"), torch.empty((T, E), device="cuda")
    idx = torch.empty((T, 2), dtype=torch.int32, device="cuda")
    m.router_topk(x.to(torch.bfloat16), w.to(torch.bfloat16), None, logits, aff, idx, m.RouterActFnType.SOFTMAX, 2, 1, 0)
    assert bool((logits == 2.0 ** 24 + 6).all())


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64, torch.int16])
def test_local_affinities_marks_what_it_cannot_refuse(dtype):
    """Ids and ranks live on the device and are not read on the host: an expert outside the table makes its token's
    affinities NaN, a rank outside it all of them; tokens without a row of ids select nothing."""
    mod = importlib.import_module("nki_library_b200.core.moe.moe_tkg.moe_tkg")
    T, E_L, E = 6, 4, 8
    aff = torch.rand((T, E), device="cuda", generator=_gen(15))
    idx = torch.tensor([[4, 5], [4, E], [-1, 6], [7, 30000], [0, 6]], device="cuda")
    if dtype == torch.int64:
        idx[3, 1] = 2 ** 32 + 5
    rank = torch.tensor([[1]], dtype=torch.int32, device="cuda")
    got = mod.local_affinities(aff, E_L, T, rank, idx.to(dtype))
    assert bool(got[1:4].isnan().all())
    want = torch.zeros((T, E_L), device="cuda")
    want[0, :2], want[4, 2] = aff[0, 4:6], aff[4, 6]
    assert torch.equal(got[[0, 4, 5]], want[[0, 4, 5]])
    assert bool(mod.local_affinities(aff, E_L, T, rank + 1, None).isnan().all())
