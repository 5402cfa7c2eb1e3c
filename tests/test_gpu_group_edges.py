"""Edges of two launches that take several things at once: a fused group repacked together with its sign and scale vectors, and routed
experts in items of up to 128 rows (an expert with one row, exactly a full item, one row more, several items; more slots than the
alignment keeps in registers), the latter against the same layer in blocks of eight rows."""
from __future__ import annotations

import pytest
import torch

from trellis_serve_b200.kernels import linear as lin
from trellis_serve_b200.kernels import moe
from trellis_serve_b200.runtime.layerset import random_signs

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _trellis(k, n, K, gen, offset=0):
    flat = torch.randint(-32768, 32767, (k // 16 * (n // 16) * 16 * K + offset,), dtype=torch.int16, device=DEV, generator=gen)
    return flat[offset:].view(k // 16, n // 16, 16 * K)


@pytest.mark.parametrize("ns", [[128], [256, 128], [128, 384, 128, 128, 256, 128, 128, 128]])
@pytest.mark.parametrize("K,offset,strided", [(2, 0, False), (3, 2, False), (8, 0, True), (5, 6, True)])
def test_group_repack_equals_its_matrices(ns, K, offset, strided):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(K)
    k = 384
    trellis = [_trellis(k, n, K, gen, offset) for n in ns]

    def vector(n):
        v = torch.randn((2 * n if strided else n + 1,), device=DEV, generator=gen).half()
        return v[::2] if strided else v[1:]

    suh, svh = [vector(k) for _ in ns], [vector(n) for n in ns]
    packed, suh_cat, svh_cat, ends = lin.prepare(trellis, suh, svh)
    assert torch.equal(packed, torch.cat([lin.prepare_matrix(t) for t in trellis]))
    assert torch.equal(suh_cat, torch.stack(suh)) and torch.equal(svh_cat, torch.cat(svh))
    assert ends == [sum(ns[:i + 1]) for i in range(len(ns) - 1)]


@pytest.mark.parametrize("rows,top_k,K,cb", [([1, 128, 129, 0], 1, 3, 0), ([700, 8, 9, 137], 1, 2, 2), ([256, 300, 255, 257], 2, 8, 1),
                                             ([6000, 5, 11000, 900], 1, 4, 0)])
def test_long_items_agree_with_blocks_of_eight(monkeypatch, rows, top_k, K, cb):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(sum(rows))
    hidden, inter, E = 384, 128, len(rows)

    def proj(k, n):
        return ([_trellis(k, n, K, gen) for _ in range(E)], [random_signs(k, gen, DEV).view(-1) for _ in range(E)],
                [(random_signs(n, gen, DEV).view(-1) / 16).half() for _ in range(E)])

    pack = moe.prepare_mixed(proj(hidden, inter), proj(hidden, inter), proj(inter, hidden), cb)
    first = torch.cat([torch.full((r,), e, dtype=torch.int32) for e, r in enumerate(rows)]).to(DEV)
    first = first[torch.randperm(first.numel(), device=DEV, generator=gen)]
    ids = torch.stack([(first + j) % E for j in range(top_k)], 1).contiguous()
    x = torch.randn((ids.shape[0], hidden), device=DEV, generator=gen).bfloat16()
    w = torch.rand(ids.shape, device=DEV, generator=gen)
    out = []
    for rows_per_expert in (0, 1 << 20):
        monkeypatch.setattr(moe, "TC_ROWS_PER_EXPERT", rows_per_expert)
        ws = torch.zeros(moe.layer_workspace_bytes([E], hidden, inter, cb, ids.shape[0], top_k), dtype=torch.uint8, device=DEV)
        y = torch.empty_like(x)
        moe.run_layer(x, w, ids, pack, y, ws)
        again = torch.empty_like(x)
        moe.run_layer(x, w, ids, pack, again, ws)
        torch.cuda.synchronize()
        assert rows_per_expert or torch.equal(y, again)      # in whatever order the alignment put the rows
        out.append(y.float())
    scale = out[1].pow(2).mean().sqrt()
    assert float((out[0] - out[1]).norm() / out[1].norm()) <= 6e-3
    assert float((out[0] - out[1]).abs().max() / scale) <= 8e-2


@pytest.mark.parametrize("rows", [65, 128, 129, 255, 257, 384, 513, 700, 1025])
@pytest.mark.parametrize("k,n,K,cb", [(384, 384, 4, 1), (1024, 1024, 2, 2)])
def test_row_tiles_that_hold_no_rows_are_left_out(rows, k, n, K, cb):
    """Many-row kernels with stale data behind the last row: the same bits as when the activation buffer was zeroed."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(rows + k)
    packed, suh_cat, svh_cat, ends = lin.prepare([_trellis(k, n, K, gen)], [random_signs(k, gen, DEV).view(-1)],
                                                 [(random_signs(n, gen, DEV).view(-1) / 16).half()])
    x = torch.randn((rows, k), device=DEV, generator=gen).half()
    need = lin.tc_workspace_bytes(rows, k, n, 1)
    out = []
    for fill in (0, 0x7F):                                   # 0x7F7F is a NaN in fp16
        ws = torch.full((need,), fill, dtype=torch.uint8, device=DEV)
        ws[:256] = 0
        y = torch.empty((rows, n), dtype=torch.float16, device=DEV)
        lin.run_tc(x, packed, suh_cat, svh_cat, ends, cb, out=y, workspace=ws)
        torch.cuda.synchronize()
        out.append(y)
    assert torch.equal(out[0], out[1]) and bool(torch.isfinite(out[0]).all())


def test_plain_calls_equal_the_operator_and_the_rest_goes_through_it():
    from trellis_serve_b200.runtime import ops

    gen = torch.Generator(device=DEV)
    gen.manual_seed(3)
    k, n, K = 256, 384, 3
    weights = lin.prepare([_trellis(k, n, K, gen)], [random_signs(k, gen, DEV).view(-1)], [(random_signs(n, gen, DEV).view(-1) / 16).half()])
    rest = ([], [], [], [], [], 0, list(weights[:3]), weights[3], [0], [n])
    op = torch.ops.exl3_b200.linear
    for x in (torch.randn((3, k), device=DEV, generator=gen).half(), torch.randn((2, 5, k), device=DEV, generator=gen), torch.zeros((0, k), device=DEV).half()):
        assert torch.equal(ops.linear(x, *rest), op(x, *rest))
        assert ops._direct(x, *rest) is not None
    assert ops._direct(x, *rest[:-1], (n,)) is None and ops._direct(x) is None          # a tuple, too few arguments
    assert torch.equal(ops.linear(x, *rest[:-1], (n,)), op(x, *rest))
    assert ops._direct(torch.nn.Parameter(x), *rest) is None
    with pytest.raises(RuntimeError, match="exceeds the stored width"):
        ops.linear(torch.zeros((1, k + 1), device=DEV), *rest)
    with torch.inference_mode():
        assert torch.equal(ops.linear(x, *rest), op(x, *rest))
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode(allow_non_fake_inputs=True):
        assert ops._direct(x, *rest) is None


def test_plain_calls_are_seen_by_whatever_watches():
    """Function modes, the profiler, gradients of any operand and tensors that are not what their storage holds: as through the operator."""
    from torch.overrides import TorchFunctionMode
    from torch.profiler import ProfilerActivity, profile

    from trellis_serve_b200.runtime import ops

    gen = torch.Generator(device=DEV)
    gen.manual_seed(4)
    k, n, K = 256, 128, 3
    packed, suh, svh, ends = lin.prepare([_trellis(k, n, K, gen)], [random_signs(k, gen, DEV).view(-1)], [(random_signs(n, gen, DEV).view(-1) / 16).half()])
    rest = ([], [], [], [], [], 0, [packed, suh, svh], ends, [0], [n])
    op = torch.ops.exl3_b200.linear
    x = torch.randn((3, k), device=DEV, generator=gen).half()
    want = op(x, *rest)

    class Watch(TorchFunctionMode):
        def __init__(self):
            super().__init__()
            self.seen = []

        def __torch_function__(self, func, types, args=(), kwargs=None):
            self.seen.append(str(func))
            return func(*args, **(kwargs or {}))

    with Watch() as watch:
        y = ops.linear(x, *rest)
        assert any("exl3_b200" in name for name in watch.seen) and ops._direct(x, *rest) is None
    assert torch.equal(y, want)
    with profile(activities=[ProfilerActivity.CPU], acc_events=True) as prof:
        y = ops.linear(x, *rest)
    assert "exl3_b200::linear" in {e.key for e in prof.key_averages()} and torch.equal(y, want)
    assert ops._direct(x, *rest) is not None                            # nothing watches any more
    learned = rest[:6] + ([packed, suh.clone().requires_grad_(), svh],) + rest[7:]
    assert ops._direct(x, *learned) is None
    with torch.no_grad():
        assert torch.equal(ops._direct(x, *learned), want)
    negated = torch._neg_view(x)
    assert torch.equal(ops.linear(negated, *rest), op(-x, *rest))
