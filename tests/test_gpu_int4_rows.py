"""int4 Linears of three to eight f32 rows (mma.sync kernel), and output matrices of few rows on the tcgen05 GEMM, against the
oracle and against each other."""
import numpy as np
import pytest

import b200nn
from b200nn import GpuTensor, synth
from oracle import oracle

pytestmark = pytest.mark.gpu


# Half a unit of 128 inputs at K's end; fewer features than a tile, a tile more; one, two and four tiles a block; K over a
# cluster (3072); groups of 128, 256 and one that K does not fill.
@pytest.mark.parametrize("m,k,n,group", [
    (3, 64, 5, 128), (8, 192, 17, 128), (7, 320, 130, 256), (8, 128, 16, 128), (5, 768, 3072, 128), (8, 3072, 768, 128),
    (4, 1600, 4800, 128), (4, 6400, 1600, 128), (8, 256, 9500, 128), (6, 320, 18000, 128)])
def test_int4_linear_of_few_rows(reg, m, k, n, group):
    packed, scales, x, _ = synth.int4_linear_case(m + k + n, m, k, n, group)
    bias = np.linspace(-1, 1, n, dtype=np.float32)
    layer = b200nn.Int4Linear(packed, scales, bias, k, n, group, reg)
    launches = reg.launch_count()
    y = layer.forward(GpuTensor.from_host(x, (m, k), reg)).to_host()
    assert reg.launch_count() - launches == 1  # no conversion of the rows
    ref = oracle.int4_linear(x, packed, scales, bias, m, n, k, group)
    rms = np.sqrt((ref ** 2).mean())
    # the rows' fp16 rounding: 2^-11 of a value at most, uniform: at most 2.8e-4 of a product on average
    assert np.sqrt(((y - ref) ** 2).mean()) / rms < 4e-4
    reg.set_tuning("int4_rows_max", 0)
    try:
        tc = layer.forward(GpuTensor.from_host(x, (m, k), reg)).to_host()  # rounds the scaled weights too
    finally:
        reg.set_tuning("int4_rows_max", -1)
    assert np.sqrt(((y - tc) ** 2).mean()) / rms < 8e-4
    x[0, 3], x[1, 5], x[2, 7] = np.inf, -np.inf, np.nan
    z = layer.forward(GpuTensor.from_host(x, (m, k), reg)).to_host()
    assert not np.isfinite(z[:3]).any() and np.array_equal(z[3:], y[3:])


# more 128-feature tiles than two blocks per SM hold, the last one ragged; one and sixteen K blocks (four small blocks per
# SM), seventeen (two larger ones)
@pytest.mark.parametrize("m,k,n", [(3, 64, 38001), (32, 1024, 38001), (17, 768, 50257), (20, 1088, 38001)])
def test_int4_output_matrix_of_few_rows(reg, m, k, n):
    packed, scales, x, _ = synth.int4_linear_case(m + k, m, k, n, 128)
    layer = b200nn.Int4Linear(packed, scales, None, k, n, 128, reg)
    y = layer.forward(GpuTensor.from_host(x, (m, k), reg)).to_host()
    ref = oracle.int4_linear(x, packed, scales, None, m, n, k, 128)
    assert np.sqrt(((y - ref) ** 2).mean()) / np.sqrt((ref ** 2).mean()) < 5e-4


# the same of a 64-row tile: its last row missing or all there, one K block, as many stages, sixteen
@pytest.mark.parametrize("m,k,n", [(33, 64, 38001), (63, 128, 38001), (64, 1024, 38001), (64, 1088, 38001)])
def test_int4_output_matrix_of_up_to_64_rows(reg, m, k, n):
    packed, scales, x, _ = synth.int4_linear_case(m + k, m, k, n, 128)
    layer = b200nn.Int4Linear(packed, scales, None, k, n, 128, reg)
    y = layer.forward(GpuTensor.from_host(x, (m, k), reg)).to_host()
    ref = oracle.int4_linear(x, packed, scales, None, m, n, k, 128)
    # rows and scaled weights rounded to fp16: 2.8e-4 of a product on average each
    assert np.sqrt(((y - ref) ** 2).mean()) / np.sqrt((ref ** 2).mean()) < 5e-4
    assert reg.device_error() == 0


def test_int4_linear_of_few_rows_at_any_address(reg):
    """Rows that start off 16 bytes take the way through the conversion kernel."""
    import torch
    packed, scales, x, _ = synth.int4_linear_case(5, 6, 256, 96, 128)
    layer = b200nn.Int4Linear(packed, scales, None, 256, 96, 128, reg)
    buf = torch.zeros(6 * 256 + 1, device="cuda")
    buf[1:] = torch.from_numpy(x).cuda().reshape(-1)
    y = torch.zeros(2, 6, 96, device="cuda")
    aligned = buf[1:].clone()
    torch.cuda.synchronize()
    layer.forward_dev(buf.data_ptr() + 4, 6, y[0].data_ptr())
    layer.forward_dev(aligned.data_ptr(), 6, y[1].data_ptr())
    reg.synchronize()
    assert y[0].abs().max() > 0 and torch.linalg.norm(y[0] - y[1]) / torch.linalg.norm(y[1]) < 8e-4


# the same buffer; results that begin in the rows' last values, and that end in their first
@pytest.mark.parametrize("k,n,at", [(256, 256, 0), (256, 96, 5 * 256 - 4), (128, 320, 4 - 5 * 320)])
def test_int4_linear_of_few_rows_over_its_own_rows(reg, k, n, at):
    """Results may lie over the rows: they are converted before the first result is stored."""
    import torch
    m = 5
    packed, scales, x, _ = synth.int4_linear_case(8, m, k, n, 128)
    layer = b200nn.Int4Linear(packed, scales, None, k, n, 128, reg)
    buf = torch.zeros(4 * m * 320, device="cuda")
    start = 2 * m * 320
    buf[start:start + m * k] = torch.from_numpy(x).cuda().reshape(-1)
    torch.cuda.synchronize()
    reg.set_tuning("int4_rows_max", 0)
    try:
        want = layer.forward(GpuTensor.from_host(x, (m, k), reg)).to_host()
    finally:
        reg.set_tuning("int4_rows_max", -1)
    launches = reg.launch_count()
    layer.forward_dev(buf.data_ptr() + 4 * start, m, buf.data_ptr() + 4 * (start + at))
    reg.synchronize()
    assert reg.launch_count() - launches == 2  # conversion, GEMM
    assert np.array_equal(buf[start + at:start + at + m * n].cpu().numpy().reshape(m, n), want)


# 64 rows of sixteen K blocks: one tile fewer and one more than two and a half per SM
@pytest.mark.parametrize("n", [370 * 128, 370 * 128 + 1])
def test_int4_output_matrix_of_64_rows_and_16_k_blocks(reg, n):
    packed, scales, x, _ = synth.int4_linear_case(7, 64, 1024, n, 128)
    layer = b200nn.Int4Linear(packed, scales, None, 1024, n, 128, reg)
    y = layer.forward(GpuTensor.from_host(x, (64, 1024), reg)).to_host()
    ref = oracle.int4_linear(x, packed, scales, None, 64, n, 1024, 128)
    # rows and scaled weights rounded to fp16: 2.8e-4 of a product on average each
    assert np.sqrt(((y - ref) ** 2).mean()) / np.sqrt((ref ** 2).mean()) < 5e-4
    assert reg.device_error() == 0


# the longest parts of K that the kernel of few rows takes with two and four tiles a block, and one unit of 128 inputs more
@pytest.mark.parametrize("m,k,n,launches", [(8, 2048, 4737, 1), (8, 2049 + 63, 4737, 2), (4, 3072, 4737, 1), (4, 3136, 4737, 2),
                                            (5, 1280, 9473, 1), (5, 1344, 9473, 2), (4, 1664, 9473, 1), (4, 1728, 9473, 2)])
def test_int4_linear_of_few_rows_stays_with_the_gemm_for_long_parts_of_k(reg, m, k, n, launches):
    packed, scales, x, _ = synth.int4_linear_case(m + k, m, k, n, 128)
    layer = b200nn.Int4Linear(packed, scales, None, k, n, 128, reg)
    before = reg.launch_count()
    y = layer.forward(GpuTensor.from_host(x, (m, k), reg)).to_host()
    assert reg.launch_count() - before == launches
    ref = oracle.int4_linear(x, packed, scales, None, m, n, k, 128)
    # rows (and, by the GEMM, scaled weights) rounded to fp16: 2.8e-4 of a product on average each
    assert np.sqrt(((y - ref) ** 2).mean()) / np.sqrt((ref ** 2).mean()) < 5e-4
