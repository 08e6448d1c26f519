"""Rows of 64 and 256 elements in the quantizer whose lanes hold 16 elements each: bit for bit the rows of the kernel with a warp per
row, which takes sources off a 16-byte boundary, and of the oracle."""
import numpy as np
import pytest
import torch

from gpu_util import TORCH_DT, fmt, pkg, words

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def P():
    return pkg()


@pytest.mark.parametrize("rotation", ["none", "hadamard"])
@pytest.mark.parametrize("dim", [64, 128, 256])
@pytest.mark.parametrize("mode,bits", [(0, 4), (0, 3), (2, 4), (3, 4), (4, 4), (5, 4)])
def test_rows_equal_those_of_a_warp_each(P, oracle, mode, bits, dim, rotation):
    qz = P.TurboQuantizer(fmt(P, mode, bits), dim, rotation, 5)
    for rows in (1, 7, 3001):
        x = torch.from_numpy(oracle.normal(70 + mode + dim, rows * dim).reshape(rows, dim)).to("cuda:0")
        x[:, :3] *= 8.0
        if rows > 7:
            x[1] = 0.0
            x[2] *= 2.0 ** -120
            x[3] = 3.0e38
            x[4, 5] = float("nan")
            x[5, 6] = float("inf")
        for name in ("f32", "f16", "bf16"):
            y = x.to(TORCH_DT[name])
            off = torch.empty(rows * dim + 1, dtype=y.dtype, device="cuda:0")[1:].view(rows, dim).copy_(y)
            got, want = words(qz.quantize_rows(y)), words(qz.quantize_rows(off))
            assert np.array_equal(got, want), f"{name}, {rows} rows: {(got != want).sum()} words differ"
            if rotation == "none":
                z = y.float().cpu().numpy()
                plain = np.isfinite(z).all(1)
                ref = oracle.quantize_rows(np.ascontiguousarray(z[plain]), mode, bits, qz.tab.cpu().numpy(), norm_order=1)
                assert np.array_equal(got[plain], ref), f"{name}, {rows} rows: {(got[plain] != ref).sum()} words differ from the oracle"
