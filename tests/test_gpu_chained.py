"""Contractions that start inside the launch in front of them read block lists, tile flags, token ids and affinities early.
Calls with very different routings follow one another on the same buffers, so that a stale word of the call before shows,
and every output is compared byte for byte with the same call on plain launches, one at a time."""

import functools

import pytest
import torch

pytestmark = pytest.mark.gpu
E, K, H, I = 24, 2, 1024, 512


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _routing(T, which):
    """[T, K] experts of token t and its affinities; every ``which`` loads other experts, and by other numbers."""
    g = _gen(100 + which)
    score = torch.rand((T, E), device="cuda", generator=g)
    score[:, which * 8:which * 8 + 5] += torch.linspace(0.9, 0.1, 5, device="cuda")
    idx = score.topk(K, dim=1).indices.to(torch.int32)
    aff = torch.zeros((T, E), device="cuda").scatter_(1, idx.long(), torch.rand((T, K), device="cuda", generator=g))
    return idx, aff


def _weights(kind):
    from nki_library_b200.layer import random_expert_weights
    from nki_library_b200.weights import prepare_dense
    if kind != "bf16":
        return random_expert_weights(E, H, I, "cuda", seed=3, w_format=5 if kind == "e2m1" else 0)
    g = _gen(3)
    return prepare_dense((torch.randn((E, H, 2, I), device="cuda", generator=g) * 0.02).to(torch.bfloat16),
                         (torch.randn((E, I, H), device="cuda", generator=g) * 0.02).to(torch.bfloat16))


def _cte(x, r, w, B):
    import nki_library_b200 as m
    idx, aff = r
    g = m.moe_group_tokens(idx, E, B, m.get_n_blocks(x.shape[0], K, E, B))
    impl = m.MoECTEImplementation.shard_on_block if hasattr(w, "scale_gu") else m.MoECTEImplementation.shard_on_block_mx
    return m.moe_cte(x, aff.view(-1, 1), w, None, g["token_position_to_id"], g["block_to_expert"], B, m.MoECTESpec(impl),
                     conditions=g["conditions"], skip_dma=m.SkipMode(True, False))


def _tkg(x, r, w, B):
    import nki_library_b200 as m
    return m.moe_tkg(x, w, None, r[1], r[0], False, expert_affinities_scaling_mode=m.ExpertAffinityScaleMode.POST_SCALE)


def _all_expert(x, r, w, B):
    import nki_library_b200 as m
    rank = torch.zeros((1, 1), dtype=torch.int32, device="cuda")
    return m.moe_tkg(x, w, None, r[1], r[0], True, rank_id=rank, mask_unselected_experts=True,
                     expert_affinities_scaling_mode=m.ExpertAffinityScaleMode.POST_SCALE)


@functools.lru_cache
def _router_w():
    return (torch.randn((H, E), device="cuda", generator=_gen(9)) * 0.05).to(torch.bfloat16)


def _block(x, r, w, B):
    import nki_library_b200 as m
    gamma = torch.ones((H,), dtype=torch.bfloat16, device="cuda")
    bias = ((r[1] > 0).float().mean(0) * 8.0).to(torch.bfloat16)  # this call routes by itself: lean on the bias
    return m.moe_block_tkg(x, gamma, _router_w(), w, None, router_bias=bias, top_k=K,
                           router_act_fn=m.RouterActFnType.SOFTMAX, norm_topk_prob=True,
                           expert_affinities_scaling_mode=m.ExpertAffinityScaleMode.POST_SCALE, is_all_expert=True,
                           rank_id=torch.zeros((1, 1), dtype=torch.int32, device="cuda"))[0]


PATHS = {"cte": (_cte, 700, 128), "cte_pair": (_cte, 700, 256), "tkg": (_tkg, 96, 128), "all_expert": (_all_expert, 96, 128),
         "block": (_block, 96, 128)}


@pytest.mark.parametrize("path,weights", [("cte", "e4m3"), ("cte_pair", "e4m3"), ("cte", "bf16"), ("cte_pair", "bf16"),
                                          ("tkg", "e4m3"), ("tkg", "e2m1"), ("tkg", "bf16"), ("all_expert", "e4m3"),
                                          ("block", "e4m3")])
@pytest.mark.parametrize("captured", [False, True])
def test_alternating_routings(path, weights, captured, monkeypatch):
    from nki_library_b200 import _lib
    fn, T, B = PATHS[path]
    w = _weights(weights)
    xs = [torch.randn((T, H), device="cuda", generator=_gen(i)).to(torch.bfloat16) for i in range(3)]
    rs = [_routing(T, i) for i in range(3)]
    ref = []
    with monkeypatch.context() as mp:
        mp.setattr(_lib, "GEMM_CHAINED", 0)
        for x, r in zip(xs, rs):
            ref.append(fn(x, r, w, B).clone())
            torch.cuda.synchronize()
    assert not torch.equal(ref[0], ref[1]) and ref[0].any()
    order = [0, 1, 2, 0, 2, 1, 0, 0, 1, 1, 2, 2]
    if not captured:
        got = [fn(xs[i], rs[i], w, B) for i in order]
    else:
        bx, br = xs[0].clone(), tuple(t.clone() for t in rs[0])
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = fn(bx, br, w, B)
        got = []
        for i in order:
            bx.copy_(xs[i])
            for b, s in zip(br, rs[i]):
                b.copy_(s)
            graph.replay()
            got.append(out.clone())
    torch.cuda.synchronize()
    for i, o in zip(order, got):
        assert torch.equal(o, ref[i])


@pytest.mark.parametrize("T,B", [(48, 128), (700, 128), (900, 256)])
@pytest.mark.parametrize("captured", [False, True])
def test_layer_alternating_routings(T, B, captured):
    from nki_library_b200.layer import MoELayer
    w = _weights("e4m3")
    rw = _router_w()
    # tokens of input i lean towards the experts of its eight columns
    xs = [(torch.randn((T, H), device="cuda", generator=_gen(i)) + 4 * rw[:, 8 * i:8 * i + 5].float().sum(1)).to(torch.bfloat16)
          for i in range(3)]
    layer = MoELayer(rw, w, K, B, T)
    ref = []
    for x in xs:
        ref.append(layer.forward(x, timers={}).clone())  # timed launch by launch: nothing is chained
        torch.cuda.synchronize()
    assert not torch.equal(ref[0], ref[1])
    order = [0, 1, 2, 0, 2, 1, 0, 0, 1, 1, 2, 2]
    got = []
    if captured:
        buf = xs[0].clone()
        layer.capture(buf)
    for i in order:
        if captured:
            buf.copy_(xs[i])
            got.append(layer.replay().clone())
        else:
            got.append(layer.forward(xs[i], out=torch.empty_like(xs[i])))
    torch.cuda.synchronize()
    assert layer.device_status() == [0, 0, 0, 0]
    for i, o in zip(order, got):
        assert torch.equal(o, ref[i])


@pytest.mark.parametrize("variant", ["single", "pair"])
def test_block_list_longer_than_the_staging_buffer(variant):
    """24 000 blocks of 128 with two tokens each: block list and flags no longer fit the shared memory they are staged in.
    Expert by expert and in scattered order, alternating, against the same tokens in full blocks (a token's row does not
    depend on where it stands)."""
    import nki_library_b200 as m
    from nki_library_b200 import _lib
    from nki_library_b200.layer import random_expert_weights
    Es, Ts, Hs, Is, N, B = 8, 6000, 128, 128, 24000, 128
    w = random_expert_weights(Es, Hs, Is, "cuda", seed=2)
    x = torch.randn((Ts, Hs), device="cuda", generator=_gen(1)).to(torch.bfloat16)
    aff = torch.rand((Ts, Es), device="cuda", generator=_gen(2))
    i32 = dict(dtype=torch.int32, device="cuda")
    impl = _lib.GEMM_NO_PAIR if variant == "single" else _lib.GEMM_FORCE_PAIR

    def run(tpi, b2e):
        return m.moe_cte(x, aff.view(-1, 1), w, None, tpi.reshape(-1), b2e, B,
                         m.MoECTESpec(m.MoECTEImplementation.shard_on_block_mx), skip_dma=m.SkipMode(True, False),
                         _impl=impl, _check_status=True)

    full = torch.full((Es, 47 * B), -1, **i32)
    full[:, :Ts] = torch.arange(Ts, **i32)
    ref = run(full, torch.arange(Es, **i32).repeat_interleave(47))
    sparse = torch.full((N, B), -1, **i32)
    sparse[:, 5] = torch.arange(Ts // 2, **i32).repeat(Es)  # not the leading rows
    sparse[:, 70] = torch.arange(Ts // 2, Ts, **i32).repeat(Es)
    b2e = torch.arange(Es, **i32).repeat_interleave(N // Es)
    perm = torch.randperm(N, device="cuda", generator=_gen(3))
    lists = [(sparse, b2e), (sparse[perm].contiguous(), b2e[perm].contiguous())]
    for i in (0, 1, 1, 0, 1):
        assert torch.equal(run(*lists[i]), ref)
