"""GPU parity of the routed-expert layer when experts see many rows each: the grouped tensor-core GEMM on 128-row moe
blocks (`exl3_moe_tc_experts`), reached through `kernels.moe.run_layer`.

The reference serves such batches by growing its moe block with T * top_k / E (cuda/src/sglang_exl3/kernels/marlin_moe.py:52-57)
and checks them with the same float64 layer reference as the decode-sized ones (tools/moe_parity_sm86.py:76-88); so do
these tests, with the oracle's np_moe_layer.  Error bars as in test_gpu_moe.py: relative L2 <= 3e-3, max|d|/rms <= 8e-3.
"""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import exl3_oracle as orc
from test_gpu_moe import _experts, _mixed_experts, _routing, _to_dev
from trellis_serve_b200.kernels import moe

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _run_layer(pack, x, w, ids, maps=None):
    tokens, top_k = ids.shape
    need = moe.layer_workspace_bytes([p.num_experts for p in pack.packs], pack.hidden, pack.inter, pack.codebook, tokens, top_k)
    ws = torch.zeros(need, dtype=torch.uint8, device=DEV)
    xt, wt, it = torch.from_numpy(x).to(DEV), torch.from_numpy(w).to(DEV), torch.from_numpy(ids).to(DEV)
    out = torch.empty_like(xt)
    moe.run_layer(xt, wt, it, pack, out, ws, maps)
    torch.cuda.synchronize()
    return out


def _check(got, ref):
    got = got.float().cpu().numpy()
    assert orc.rel_norm(got, ref) <= 3e-3, orc.rel_norm(got, ref)
    assert orc.max_over_rms(got, ref) <= 8e-3, orc.max_over_rms(got, ref)


@pytest.mark.parametrize("tokens,E,zipf", [(300, 8, False), (700, 4, True), (130, 8, True)])
@pytest.mark.parametrize("K,cb", [(3, 0), (4, 1), (3, 2)])
def test_many_rows_per_expert_match_the_float64_reference(tokens, E, zipf, K, cb):
    """75, 350 and 32 rows per expert on average: single blocks with padding, experts of several 128-row blocks (work items of
    up to four blocks, more than one item for the heavy experts under zipf routing) and experts with no rows at all."""
    hidden, inter, top_k = 256, 128, 2
    assert moe.moe_block_size(tokens, top_k, E) == 128
    gate, up, down = _experts(500 * K + cb + E, E, hidden, inter, K, out_scale=1 / 8)
    pack = moe.prepare_mixed(_to_dev(gate), _to_dev(up), _to_dev(down), cb)
    ids, w = _routing(tokens, top_k, E, 11 + tokens, zipf)
    ids[0, 0] = -1                                                             # an invalid id is dropped, not routed
    x = np.random.default_rng(tokens).standard_normal((tokens, hidden)).astype(np.float16)
    _check(_run_layer(pack, x, w, ids), orc.np_moe_layer(x, ids, w, gate, up, down, K, cb))


def test_tensor_core_and_decode_paths_agree_and_bf16_boundary(monkeypatch):
    """The same batch through both paths: they differ only by fp16 roundings of intermediates.  bf16 in / out equals explicit casts."""
    E, hidden, inter, top_k, K, cb, tokens = 8, 512, 256, 2, 4, 1, 200
    gate, up, down = _experts(909, E, hidden, inter, K, out_scale=1 / 16)
    pack = moe.prepare_mixed(_to_dev(gate), _to_dev(up), _to_dev(down), cb)
    ids, w = _routing(tokens, top_k, E, 5)
    x = np.random.default_rng(1).standard_normal((tokens, hidden)).astype(np.float16)
    tc = _run_layer(pack, x, w, ids)
    monkeypatch.setattr(moe, "TC_ROWS_PER_EXPERT", 1 << 30)
    assert moe.moe_block_size(tokens, top_k, E) == 8
    gemv = _run_layer(pack, x, w, ids)
    monkeypatch.undo()
    assert orc.rel_norm(tc.float().cpu().numpy(), gemv.float().cpu().numpy()) <= 2e-3
    _check(tc, orc.np_moe_layer(x, ids, w, gate, up, down, K, cb))
    xb = torch.from_numpy(x).to(DEV).bfloat16()
    need = moe.layer_workspace_bytes([E], hidden, inter, cb, tokens, top_k)
    ws = torch.zeros(need, dtype=torch.uint8, device=DEV)
    outb = torch.empty_like(xb)
    moe.run_layer(xb, torch.from_numpy(w).to(DEV), torch.from_numpy(ids).to(DEV), pack, outb, ws)
    via_half = _run_layer(pack, xb.half().cpu().numpy(), w, ids)
    assert torch.equal(outb, via_half.bfloat16())


def test_mixed_bitrate_and_expert_map_with_many_rows():
    """Two bitrate classes, both above the switch; then an engine-style expert map that leaves experts 1 and 6 to another rank:
    their slots add nothing."""
    Ks = [3, 4, 3, 3, 4, 3, 4, 3]
    E, hidden, inter, top_k, cb, tokens = len(Ks), 256, 128, 2, 0, 400
    gate, up, down = _mixed_experts(7100, Ks, hidden, inter)
    for proj in (gate, up, down):
        proj[2][:] = [(s.astype(np.float32) / 8).astype(np.float16) for s in proj[2]]
    pack = moe.prepare_mixed(_to_dev(gate), _to_dev(up), _to_dev(down), cb)
    assert all(moe.moe_block_size(tokens, top_k, p.num_experts) == 128 for p in pack.packs)
    ids, w = _routing(tokens, top_k, E, 77, zipf=True)
    x = np.random.default_rng(2).standard_normal((tokens, hidden)).astype(np.float16)
    _check(_run_layer(pack, x, w, ids), orc.np_moe_layer(x, ids, w, gate, up, down, Ks, cb))
    held = [e for e in range(E) if e not in (1, 6)]
    maps = []
    for m in pack.expert_maps:
        m2 = m.clone()
        m2[[1, 6]] = -1
        maps.append(m2)
    ids_held = np.where(np.isin(ids, held), ids, -1)
    _check(_run_layer(pack, x, w, ids, maps), orc.np_moe_layer(x, ids_held, w, gate, up, down, Ks, cb))


def test_graph_replay_with_fresh_routing_allocates_nothing():
    E, hidden, inter, top_k, K, cb, tokens = 4, 256, 128, 2, 3, 0, 160
    gate, up, down = _experts(31, E, hidden, inter, K, out_scale=1 / 8)
    pack = moe.prepare_mixed(_to_dev(gate), _to_dev(up), _to_dev(down), cb)
    need = moe.layer_workspace_bytes([E], hidden, inter, cb, tokens, top_k)
    ws = torch.zeros(need, dtype=torch.uint8, device=DEV)
    ids, w = _routing(tokens, top_k, E, 1)
    xs = torch.randn((tokens, hidden), device=DEV).half()
    wt, it = torch.from_numpy(w).to(DEV), torch.from_numpy(ids).to(DEV)
    out, out2 = torch.empty_like(xs), torch.empty_like(xs)
    moe.run_layer(xs, wt, it, pack, out, ws)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    moe.run_layer(xs, wt, it, pack, out2, ws)
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() == before and torch.equal(out, out2)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        moe.run_layer(xs, wt, it, pack, out, ws)
    ids2, w2 = _routing(tokens, top_k, E, 2, zipf=True)
    x2 = torch.randn((tokens, hidden), device=DEV).half()
    moe.run_layer(x2, torch.from_numpy(w2).to(DEV), torch.from_numpy(ids2).to(DEV), pack, out2, ws)
    xs.copy_(x2)
    wt.copy_(torch.from_numpy(w2).to(DEV))
    it.copy_(torch.from_numpy(ids2).to(DEV))
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, out2)


@pytest.mark.parametrize("top_k,tokens,dtype", [(1, 90, torch.float16), (2, 61, torch.bfloat16), (3, 57, torch.float16), (5, 33, torch.bfloat16),
                                               (8, 30, torch.float16), (11, 17, torch.bfloat16)])
def test_last_rotation_and_sum_in_one_launch(top_k, tokens, dtype):
    """exl3_moe_tc_layer against exl3_moe_tc_experts + exl3_moe_combine, which an output that is not 16-byte aligned takes: the same roundings
    of the slots' rows, their fp32 sum in another order -- at most a unit in the last place of the result, and at 2^-22 of the summed values
    in all.  Top-k from one to more than a warp's eight rows, tokens that do not fill the last warp, ids out of range and an expert that
    the map leaves out."""
    E, hidden, inter, K, cb = 12 if top_k == 11 else 8, 384, 128, 3, 0
    gate, up, down = _experts(51 + top_k, E, hidden, inter, K, out_scale=1 / 8)
    pack = moe.prepare_mixed(_to_dev(gate), _to_dev(up), _to_dev(down), cb)
    assert moe.moe_block_size(tokens, top_k, E) == 128
    ids, w = _routing(tokens, top_k, E, 5 + top_k)
    ids[0, 0], ids[1, 0] = -1, E
    emap = pack.expert_maps[0].clone()
    emap[3] = -1
    x = torch.randn((tokens, hidden), device=DEV, generator=torch.Generator(device=DEV).manual_seed(2)).to(dtype)
    wt, it = torch.from_numpy(w).to(DEV), torch.from_numpy(ids).to(DEV)
    ws = torch.zeros(moe.layer_workspace_bytes([E], hidden, inter, cb, tokens, top_k), dtype=torch.uint8, device=DEV)
    one, again = torch.empty_like(x), torch.empty_like(x)
    two = torch.empty(tokens * hidden + 2, dtype=dtype, device=DEV)[2:].view(tokens, hidden)
    for maps in (None, [emap]):
        for out in (one, again, two):
            moe.run_layer(x, wt, it, pack, out, ws, maps)
        torch.cuda.synchronize()
        assert torch.equal(one, again)
        ulp = 2.0 ** -10 if dtype == torch.float16 else 2.0 ** -7
        a, b = one.float(), two.float()
        assert bool(((a - b).abs() <= ulp * b.abs() + 2.0 ** -22 * b.abs().max()).all())
        assert float((a != b).float().mean()) <= 0.02


@pytest.mark.parametrize("hidden,inter", [(640, 384), (128, 128), (1152, 256)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_rotations_of_pairs_of_row_blocks(hidden, inter, dtype):
    """The rotations take two neighbouring blocks of eight rows or two column blocks at a time: experts with one row, exactly one block, an odd
    and an even number of blocks and more than an item's 128 rows, so that pairs lie within an item, across two and at the end; odd numbers of
    column blocks, and one alone.  fp16: the bars of this file; bf16 adds the rounding of the result, 2^-9 of a value."""
    K, cb, E = 3, 0, 6
    counts = [1, 8, 24, 9, 133, 17]
    gate, up, down = _experts(77 + hidden, E, hidden, inter, K, out_scale=1 / 8)
    pack = moe.prepare_mixed(_to_dev(gate), _to_dev(up), _to_dev(down), cb)
    rng = np.random.default_rng(hidden)
    ids = rng.permutation(np.repeat(np.arange(E), counts)).astype(np.int32)[:, None]
    tokens = len(ids)
    assert moe.moe_block_size(tokens, 1, E) == 128
    w = rng.uniform(0.5, 1.0, (tokens, 1)).astype(np.float32)
    x = rng.standard_normal((tokens, hidden)).astype(np.float16)
    xt = torch.from_numpy(x).to(DEV).to(dtype)
    ref = orc.np_moe_layer(xt.to(torch.float16).cpu().numpy(), ids, w, gate, up, down, K, cb)
    ws = torch.zeros(moe.layer_workspace_bytes([E], hidden, inter, cb, tokens, 1), dtype=torch.uint8, device=DEV)
    out = torch.empty_like(xt)
    moe.run_layer(xt, torch.from_numpy(w).to(DEV), torch.from_numpy(ids).to(DEV), pack, out, ws, None)
    got = out.float().cpu().numpy()
    if dtype == torch.float16:
        _check(out, ref)
    else:
        assert orc.rel_norm(got, ref) <= 3e-3 + 2.0 ** -9


@pytest.mark.parametrize("K,cb", [(6, 0), (7, 1), (8, 2), (8, 0)])
def test_long_items_at_high_bit_rates(K, cb):
    """Three stages of three units leave the activations of 128 rows three slots of shared memory at 6 and 7 bits and two at 8: items of all 128 rows,
    of few and of 64, six units deep, so that both rings are lapped many times (the bars of this file)."""
    hidden, inter, E = 768, 640, 5
    gate, up, down = _experts(7 * K + cb, E, hidden, inter, K, out_scale=1 / 8)
    pack = moe.prepare_mixed(_to_dev(gate), _to_dev(up), _to_dev(down), cb)
    rng = np.random.default_rng(K)
    ids = rng.permutation(np.repeat(np.arange(E), [300, 128, 64, 3, 17])).astype(np.int32)[:, None]
    assert moe.moe_block_size(len(ids), 1, E) == 128
    w = rng.uniform(0.5, 1.0, ids.shape).astype(np.float32)
    x = rng.standard_normal((len(ids), hidden)).astype(np.float16)
    _check(_run_layer(pack, x, w, ids), orc.np_moe_layer(x, ids, w, gate, up, down, K, cb))
