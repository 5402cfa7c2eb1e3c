"""The rotations that run on tensor cores, sixteen rows at a time: each row against float64, beside rows of other magnitudes and rows that are not
finite."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import exl3_oracle as orc
from test_gpu_moe import _experts, _to_dev
from trellis_serve_b200.kernels import linear as lin
from trellis_serve_b200.kernels import moe
from trellis_serve_b200.runtime.layerset import random_packed, random_signs

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _had128(n: int) -> torch.Tensor:
    h = torch.ones((1, 1), dtype=torch.float64, device=DEV)
    while h.shape[0] < 128:
        h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)], 0)
    return h


def _operand(ws: torch.Tensor, rows: int, k: int) -> torch.Tensor:
    """The rotated rows that the many-row product left in its workspace: super tiles of 512 rows x 64 columns, in them 128 rows x chunks of eight
    columns x blocks of eight rows."""
    tiles = (rows + 511) // 512
    a = ws[256:256 + tiles * 512 * k * 2].view(torch.float16).view(tiles, k // 64, 4, 8, 16, 8, 8)     # tile, k block, 128 rows, chunk, block, row, column
    return a.permute(0, 2, 4, 5, 1, 3, 6).reshape(tiles * 512, k)[:rows]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows", [65, 97, 128, 520])
def test_rows_of_the_many_row_product(rows, dtype):
    """A result is the fp32 sum of 128 exact products, rounded to fp16: half a unit in the last place (2^-11 of the value, 2^-25 below the normal
    numbers) plus the sum's own error -- sixteen additions in the tensor core, three of butterflies and the scale, each off by at most 2^-23 of
    the sum of the magnitudes."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(rows)
    k, n = 384, 256
    x = torch.randn((rows, k), device=DEV, generator=gen)
    x *= torch.tensor([1.0, 1e-4, 5e3], device=DEV)[torch.arange(rows, device=DEV) % 3][:, None]
    x = x.to(dtype)
    bad = {7: float("inf"), 18: float("nan"), 30: float("-inf"), rows - 1: float("nan")}
    for row, value in bad.items():
        x[row, 130] = value                                  # of the second block of 128 columns
    suh = (random_signs(k, gen, DEV).view(-1) * (1 + 0.1 * torch.randn(k, device=DEV, generator=gen))).half()
    packed, svh = random_packed(k, n, 3, gen, DEV), random_signs(n, gen, DEV).view(-1)
    ws = torch.zeros(lin.tc_workspace_bytes(rows, k, n, 1), dtype=torch.uint8, device=DEV)
    y = lin.run_tc(x, packed, suh, svh, [], 0, workspace=ws)
    torch.cuda.synchronize()
    got = _operand(ws, rows, k).double()
    terms = (x.half().double() * suh.double()).view(rows, -1, 128)
    want = (terms @ _had128(128)).reshape(rows, k) / 128 ** 0.5
    size = (terms.abs().sum(-1, keepdim=True) / 128 ** 0.5).expand_as(terms).reshape(rows, k)
    clean = torch.ones((rows, k), dtype=torch.bool, device=DEV)
    for row in bad:
        clean[row, 128:256] = False
    assert not bool(torch.isfinite(got[~clean]).any())
    assert bool(torch.isfinite(got[clean]).all())
    bound = want.abs() * 2.0 ** -11 + 2.0 ** -25 + 20 * 2.0 ** -23 * size
    assert bool(((got - want).abs()[clean] <= bound[clean]).all())
    keep = torch.tensor([r for r in range(rows) if r not in bad], device=DEV)
    alone = x.clone()
    alone[list(bad)] = 0
    bits = [t[keep].view(torch.int16) for t in (y, lin.run_tc(alone, packed, suh, svh, [], 0))]      # sums of the largest rows are beyond fp16
    assert torch.equal(*bits)


@pytest.mark.parametrize("top_k", [1, 2, 3])
def test_rows_of_routed_experts(top_k):
    """Rows a hundred times apart in size, each against the float64 layer (the bar of the other tests, which hold it over whole batches: 3e-3), and
    the same bits beside tokens that are not finite."""
    hidden, inter, K, cb, E, tokens = 384, 256, 4, 1, 4, 120
    gate, up, down = _experts(31 + top_k, E, hidden, inter, K, out_scale=1 / 8)
    pack = moe.prepare_mixed(_to_dev(gate), _to_dev(up), _to_dev(down), cb)
    assert moe.moe_block_size(tokens, top_k, E) == 128
    rng = np.random.default_rng(top_k)
    ids = np.stack([rng.permutation(E)[:top_k] for _ in range(tokens)]).astype(np.int32)
    w = rng.uniform(0.5, 1.0, (tokens, top_k)).astype(np.float32)
    x = (rng.standard_normal((tokens, hidden)) * np.array([0.1, 1.0, 10.0])[np.arange(tokens) % 3][:, None]).astype(np.float16)
    ref = orc.np_moe_layer(x, ids, w, gate, up, down, K, cb)

    def run(x):
        ws = torch.zeros(moe.layer_workspace_bytes([E], hidden, inter, cb, tokens, top_k), dtype=torch.uint8, device=DEV)
        xt = torch.from_numpy(x).to(DEV)
        out = torch.empty_like(xt)
        moe.run_layer(xt, torch.from_numpy(w).to(DEV), torch.from_numpy(ids).to(DEV), pack, out, ws, None)
        torch.cuda.synchronize()
        return out

    y = run(x)
    got = y.double().cpu().numpy()
    finite = np.isfinite(got).all(axis=1)                    # silu(gate) * up of the largest rows may be beyond fp16
    assert finite[np.arange(tokens) % 3 < 2].all() and finite.mean() > 0.9
    assert float((np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1))[finite].max()) <= 3e-3
    bad = x.copy()
    bad[[3, 40, 119], 5] = np.inf, np.nan, -np.inf
    keep = torch.tensor([t for t in range(tokens) if t not in (3, 40, 119)], device=DEV)
    beside = run(bad)
    assert torch.equal(beside[keep].view(torch.int16), y[keep].view(torch.int16))
    assert not bool(torch.isfinite(beside[3]).any())
