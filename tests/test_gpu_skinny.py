"""The decode GEMV / skinny GEMM at the edges of its row pitches (1-2, 3-8, 9-16, 17-32, 33-64 rows) and of its stage ring (ranges of
one unit, ranges that wrap the ring several times), with and without the rotation inside, against a plain fp32 product on the decoded
weights."""
from __future__ import annotations

import ctypes

import pytest
import torch

from trellis_serve_b200.kernels import linear as lin
from trellis_serve_b200.runtime.layerset import random_packed, random_signs

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _had128(x: torch.Tensor) -> torch.Tensor:
    h = torch.ones((1, 1), device=x.device)
    while h.shape[0] < 128:
        h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)], 0)
    return (x.view(x.shape[0], -1, 128) @ (h / 128 ** 0.5)).reshape(x.shape)


@pytest.mark.parametrize("rows", [1, 2, 3, 8, 9, 16, 17, 32, 33, 64, 65])
@pytest.mark.parametrize("k,ns,K,cb", [(128, [128], 3, 0), (384, [256, 128], 8, 1), (5120, [5120, 1024, 1024], 3, 0), (17408, [2048], 2, 2),
                                       (2176, [17408], 8, 0), (5120, [10240], 5, 1)])
def test_rows_and_ring_edges(rows, k, ns, K, cb):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(rows + k)
    packed = torch.cat([random_packed(k, n, K, gen, DEV) for n in ns])
    suh, svh = random_signs(k, gen, DEV, len(ns)), (random_signs(sum(ns), gen, DEV).view(-1) / 64).half()
    ends = [sum(ns[:i + 1]) for i in range(len(ns) - 1)]
    dtype = torch.bfloat16 if rows % 2 else torch.float16
    x = torch.randn((rows, k), device=DEV, generator=gen).to(dtype)
    y = torch.empty((rows, sum(ns)), dtype=torch.float32, device=DEV)
    lin.run(x, packed, suh, svh, ends, cb, out=y)
    again = torch.empty_like(y)
    lin.run(x, packed, suh, svh, ends, cb, out=again)
    torch.cuda.synchronize()
    lin.device_error(DEV)
    assert torch.equal(y, again)
    xh = lin.had_in_group(x, suh).float()
    col = 0
    torch.backends.cuda.matmul.allow_tf32 = False
    for s, n in enumerate(ns):
        w = lin.reconstruct_packed(packed[col // 128:(col + n) // 128].contiguous(), cb).float()
        want = _had128(xh[s * rows:(s + 1) * rows] @ w) * svh[col:col + n].float()
        got = y[:, col:col + n]
        assert float((got - want).norm() / want.norm()) <= 1e-3
        assert float((got - want).abs().max() / want.pow(2).mean().sqrt()) <= 2e-3
        col += n


@pytest.mark.parametrize("rows", [1, 9, 57, 65, 130])
@pytest.mark.parametrize("x_cols,widths", [(1000, [1000, 130]), (1021, [128, 1]), (8, [7, 256]), (1024, [900, 255])])
def test_true_sizes_below_the_stored_ones(rows, x_cols, widths):
    from trellis_serve_b200.runtime import ops

    gen = torch.Generator(device=DEV)
    gen.manual_seed(rows * 7 + x_cols)
    k, K = 1024, 4
    ns = [(w + 127) // 128 * 128 for w in widths]
    trellis = [torch.randint(-32768, 32767, (k // 16, n // 16, 16 * K), dtype=torch.int16, device=DEV, generator=gen) for n in ns]
    suh = [random_signs(k, gen, DEV, 1).view(-1) for _ in ns]
    svh = [(random_signs(n, gen, DEV).view(-1) / 64).half() for n in ns]
    x = torch.randn((rows, x_cols), device=DEV, generator=gen).half()
    padded = torch.nn.functional.pad(x, (0, k - x_cols))
    packed, suh_cat, svh_cat, ends = lin.prepare(trellis, suh, svh)
    whole = ops.linear(padded, [], [], [], [], [], 0, [packed, suh_cat, svh_cat], ends, [0, 0], ns)
    got = ops.linear(x, [], [], [], [], [], 0, [packed, suh_cat, svh_cat], ends, [0, 0], widths)
    torch.cuda.synchronize()
    lin.device_error(DEV)
    want = torch.cat([whole[:, sum(ns[:i]):sum(ns[:i]) + w] for i, w in enumerate(widths)], 1)
    assert torch.equal(got, want)


@pytest.mark.parametrize("rows", [1, 5, 16, 40])
@pytest.mark.parametrize("k,n,K,cb", [
    (1024, 640, 3, 0),          # a unit per CTA
    (1280, 5120, 4, 1),         # three parts of three and four units; whole column blocks from nine rows up
    (896, 4736, 2, 2),          # a column block per CTA, 37 CTAs
    (128, 19200, 8, 0),         # one unit deep, 150 column blocks: two for two of the CTAs
    (512, 38016, 5, 1),         # 297 column blocks of four units: two or three per CTA
    (9600, 512, 3, 0),          # 37 parts of two and three units
    (16384, 256, 6, 2),         # 74 parts
])
def test_column_blocks_and_parts_of_them(rows, k, n, K, cb):
    """The ways of dealing units to CTAs other than even ranges: whole column blocks, equal parts of one, remainders of both, against a plain
    fp32 product on the decoded weights (bounds of the test above)."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(rows + n)
    packed, suh, svh = random_packed(k, n, K, gen, DEV), random_signs(k, gen, DEV, 1), (random_signs(n, gen, DEV).view(-1) / 64).half()
    x = torch.randn((rows, k), device=DEV, generator=gen).half()
    y, again = (torch.empty((rows, n), dtype=torch.float32, device=DEV) for _ in range(2))
    lin.run(x, packed, suh, svh, [], cb, out=y)
    lin.run(x, packed, suh, svh, [], cb, out=again)
    torch.cuda.synchronize()
    lin.device_error(DEV)
    assert torch.equal(y, again)
    torch.backends.cuda.matmul.allow_tf32 = False
    want = _had128(lin.had_in_group(x, suh).float() @ lin.reconstruct_packed(packed, cb).float()) * svh.float()
    assert float((y - want).norm() / want.norm()) <= 1e-3
    assert float((y - want).abs().max() / want.pow(2).mean().sqrt()) <= 2e-3


@pytest.mark.parametrize("rows,k,n,K,cb", [
    (1, 8576, 36864, 3, 0),     # 134 units in whole column blocks, 131 in even ranges
    (2, 10368, 36992, 3, 2),    # 162 and 159
    (5, 1024, 47488, 8, 0),     # 24 and 21
    (8, 896, 46080, 8, 1),      # 21 and 18
])
def test_even_ranges_where_the_rows_of_whole_column_blocks_do_not_fit(rows, k, n, K, cb):
    """Sizes for which whole column blocks cost less but the busiest CTA's rotated and raw rows (1792 bytes a unit for two rows split, 6400 for
    eight) leave no room for a ring of stages in 227 KB, while those of even ranges do."""
    test_column_blocks_and_parts_of_them(rows, k, n, K, cb)


def _launches(call):
    """Kernels that `call` launches: the nodes of its captured graph."""
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    count = ctypes.c_size_t(0)
    assert ctypes.CDLL("libcuda.so.1").cuGraphGetNodes(ctypes.c_void_p(graph.raw_cuda_graph()), None, ctypes.byref(count)) == 0
    return count.value


@pytest.mark.parametrize("rows,k,n,K,cb,launches", [
    (1, 5120, 34816, 8, 0, 1),      # 74 units per CTA: a ring of two stages of three units, 96 KB
    (2, 5120, 34816, 8, 2, 1),      # the same beside two rows of paired weights
    (1, 5120, 34816, 7, 0, 2),      # two of three would hold 84 KB
    (2, 5120, 34816, 6, 0, 2),      # ... 72 KB
    (2, 5120, 34816, 8, 0, 2),      # two do not fit
    (1, 8576, 36864, 3, 0, 2),      # neither do they in even ranges of 131 units
    (2, 6272, 36352, 3, 0, 1),      # 98 units in whole column blocks do not fit, 95 in even ranges do: three stages of three
    (1, 5504, 36224, 8, 0, 1),      # 86 and 83: two of three
    (2, 4736, 35968, 8, 0, 1),      # 74 and 71: two of three
])
def test_rings_of_long_ranges(rows, k, n, K, cb, launches):
    """One or two rows over ranges that leave room for few stages: the smallest rings, many laps of them, even ranges where whole column blocks
    do not fit, and the lines beyond which a launch of its own rotates the rows."""
    test_column_blocks_and_parts_of_them(rows, k, n, K, cb)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(1)
    packed, suh, svh = random_packed(k, n, K, gen, DEV), random_signs(k, gen, DEV, 1), random_signs(n, gen, DEV).view(-1)
    x, y = torch.randn((rows, k), device=DEV, generator=gen).half(), torch.empty((rows, n), dtype=torch.float16, device=DEV)
    ws = torch.zeros(lin.workspace_bytes(rows, k, n, 1), dtype=torch.uint8, device=DEV)
    assert _launches(lambda: lin.run(x, packed, suh, svh, [], cb, out=y, workspace=ws)) == launches


@pytest.mark.parametrize("rows,K,cb,launches", [(1, 3, 0, 1), (2, 5, 0, 2), (1, 6, 0, 2), (2, 7, 2, 2), (1, 8, 2, 1), (2, 8, 0, 2)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_rings_of_long_ranges_normalised(rows, K, cb, launches, dtype):
    """The normalising form beside 74 units per CTA, on either side of the line, against the normalisation on its own and a plain linear: they
    differ by the last bit of the normalisation factor, which flips the rounding of an activation here and there (the bar of the decode step's
    tests for the same pair)."""
    k, n = 5120, 34816
    gen = torch.Generator(device=DEV)
    gen.manual_seed(rows + K)
    packed, suh, svh = random_packed(k, n, K, gen, DEV), random_signs(k, gen, DEV, 2), (random_signs(n, gen, DEV).view(-1) / 64).half()
    z = torch.randn((rows, k), device=DEV, generator=gen).to(dtype)
    weight = (1.0 + 0.1 * torch.randn(k, device=DEV, generator=gen)).to(dtype)
    ssq = z.float().view(rows, k // 128, 128).pow(2).sum(-1).contiguous()
    got, act = torch.empty((rows, n), dtype=torch.float32, device=DEV), torch.empty_like(z)
    ws = torch.zeros(lin.workspace_bytes(rows, k, n, 2), dtype=torch.uint8, device=DEV)
    assert _launches(lambda: lin.run_normed(z, ssq, weight, 1e-6, packed, suh, svh, [n // 2], cb, got, ws)) == launches
    got.zero_()
    lin.run_normed(z, ssq, weight, 1e-6, packed, suh, svh, [n // 2], cb, got, ws)
    lin.normed(z, ssq, weight, 1e-6, act)
    want = lin.run(act, packed, suh, svh, [n // 2], cb, out=torch.empty_like(got))
    torch.cuda.synchronize()
    lin.device_error(DEV)
    scale = float(want.pow(2).mean().sqrt())
    assert float((got - want).abs().max()) <= 2e-3 * scale * (1 if dtype == torch.float16 else 8)      # bf16 activations: eight times the step
