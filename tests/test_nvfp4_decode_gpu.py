"""The tcgen05 kernel of few-row NVFP4 linears (csrc/nvfp4_decode.cuh) where it can go wrong: K below, at and past its unit of 256
and past a cluster's share, output rows that end inside a tile, row counts at the edges of a launch, and activations whose
magnitudes one grid cannot cover."""

import numpy as np
import pytest

from oracle import oracle_c as OC
from oracle import oracle_np as O
from tests.gpu_util import Device, random_x

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    device = Device()
    yield device
    assert device.gpu.take_device_error() == 0
    device.release()


def run(dev, x_bits, d_w, n, k, size):
    rows = x_bits.shape[0]
    d_x, d_y = dev.put(x_bits), dev.empty(rows * n * 2)
    with dev.submit(pdl=True, row_exact=True) as gpu:
        gpu.linear_nvfp4_bf16(d_x.data_ptr(), d_w.data_ptr(), d_y.data_ptr(), rows, k, n, size)
    return dev.get(d_y, np.uint16, (rows, n))


@pytest.mark.parametrize("n,k", [(16, 128), (144, 256), (112, 384), (272, 1152), (1040, 4224), (128, 12416)])
def test_edges_and_outliers(dev, n, k):
    rng = np.random.default_rng(n + k)
    weights = (rng.standard_normal((n, k)) * 0.02).astype(np.float32)
    weights[:, 5::97] *= rng.integers(0, 2, (n, len(range(5, k, 97))))     # half of the outliers meet a zero weight
    blob = OC.nvfp4_quantize(weights)
    dense = OC.nvfp4_dense(blob, n, k)
    d_w = dev.put(blob)
    plain = rng.standard_normal((17, k)).astype(np.float32)
    wide = plain.copy()
    wide[:, 5::97] *= np.float32(2.0) ** rng.integers(4, 14, wide[:, 5::97].shape)   # up to 2^13 of their neighbours
    wide[3] = plain[3]                                                             # rows of both kinds side by side
    wide[4, : k // 2] = 0.0
    wide[5] *= np.float32(2.0) ** -60
    for values in (plain, wide):
        x = O.bf16_bits(values)
        single = np.concatenate([run(dev, x[r:r + 1], d_w, n, k, blob.size) for r in range(6)])
        for rows in (2, 7, 16, 17):
            got_bits = run(dev, x[:rows], d_w, n, k, blob.size)
            assert np.array_equal(got_bits[:6], single[:min(rows, 6)]), rows          # a row's bits are its own
            got, expect = O.bf16_to_f32(got_bits).astype(np.float64), O.linear_f64(x[:rows], dense)
            # half a BF16 step of the value, and the rounding of FP32 sums of the terms that it is made of
            terms = np.abs(O.bf16_to_f32(x[:rows]).astype(np.float64)) @ np.abs(dense.astype(np.float64)).T
            assert np.all(np.abs(got - expect) <= np.abs(expect) * 2.0 ** -8 + terms * 2.0 ** -18), (rows, n, k)


def test_few_and_many_exchange_buffers(dev):
    """16 rows of K = 5376 leave room for two exchange buffers beside the digits, one row for four: several tiles per cluster, so that
    both sets are used again, give a row the same bits."""
    from euhedral_b200 import synthetic
    n, k = 18944, 5376                                            # four tiles of 128 rows for each of 37 clusters
    d_w = synthetic.nvfp4_tensor(synthetic.gaussian(n, k, 5, 0.02, device="cuda"))
    x = random_x(np.random.default_rng(6), 16, k)
    for _ in range(3):
        got = run(dev, x, d_w, n, k, d_w.numel())
        for row in (0, 7, 15):
            assert np.array_equal(run(dev, x[row:row + 1], d_w, n, k, d_w.numel())[0], got[row]), row


@pytest.mark.parametrize("n,k", [(48, 384), (160, 5120), (32, 69632)])     # the last: more than 32 units of K in a CTA
@pytest.mark.parametrize("sd4", [False, True])
def test_every_finite_value_counts(dev, n, k, sd4):
    """Outputs whose weights are zero wherever the activations are large: what is left must count in full, however far below the
    row's largest value it lies."""
    rng = np.random.default_rng(n + k + sd4)
    x = rng.standard_normal((9, k))
    x[1, 7] = 2.0 ** 100                                          # one value that no common grid spans with the others
    x[2] *= 2.0 ** rng.integers(-60, 60, k)                       # all over
    x[3] *= 2.0 ** -112                                           # next to nothing
    x[4, : k // 2] *= 2.0 ** -17                                  # two populations inside a slice
    x[5, ::3] = 0.0
    x[6] = np.where(np.arange(k) % 97 == 5, 2.0 ** 90, 2.0 ** -90)
    x[7] = 0.0
    x[8, ::50] *= 2.0 ** 14
    x = O.bf16_bits(x.astype(np.float32))
    values = O.bf16_to_f32(x).astype(np.float64)
    weights = (rng.standard_normal((n, k)) * 0.02).astype(np.float32)
    for j in range(n):                                            # weight row j sees the smallest (j + 1) / n of row j % 9
        size = np.abs(values[j % 9])
        weights[j, size > np.quantile(size, (j + 1) / n)] = 0.0
    weights[0, np.argsort(np.abs(values[0]))[3:]] = 0.0           # and the first of them three values
    blob = OC.nvfp4_quantize(weights).tobytes()
    if sd4:
        blob = O.nvfp4_sd4_from_plain(blob, n, k, rng)
    dense = O.nvfp4_dense(O.nvfp4_sd4_to_plain(blob, n, k) if sd4 else blob, n, k).astype(np.float64)
    d_w = dev.put(np.frombuffer(blob, dtype=np.uint8))
    got_bits = run(dev, x, d_w, n, k, len(blob))
    got, expect, terms = O.bf16_to_f32(got_bits).astype(np.float64), values @ dense.T, np.abs(values) @ np.abs(dense).T
    assert np.all(np.abs(got - expect) <= np.abs(expect) * 2.0 ** -8 + terms * 2.0 ** -18)   # half a BF16 step and rounded FP32 sums
    for row in range(9):
        assert np.array_equal(run(dev, x[row:row + 1], d_w, n, k, len(blob))[0], got_bits[row]), row


@pytest.mark.parametrize("n,k", [(64, 512), (144, 1152), (272, 5120)])
@pytest.mark.parametrize("sd4", [False, True])
def test_values_that_are_not_finite(dev, n, k, sd4):
    """An infinity gives every output of its row an infinity of the product's sign, NaN where it meets a zero weight or an infinity of
    the other sign; a NaN makes its row NaN. Rows without such values keep their bits."""
    rng = np.random.default_rng(n + k)
    weights = (rng.standard_normal((n, k)) * 0.02).astype(np.float32)
    weights[::3, 300] = weights[1::5, 17] = 0.0
    blob = OC.nvfp4_quantize(weights).tobytes()
    if sd4:
        blob = O.nvfp4_sd4_from_plain(blob, n, k, rng)
    dense = O.nvfp4_dense(O.nvfp4_sd4_to_plain(blob, n, k) if sd4 else blob, n, k)
    d_w = dev.put(np.frombuffer(blob, dtype=np.uint8))
    x = random_x(rng, 7, k)
    clean = run(dev, x, d_w, n, k, len(blob))
    x[1, 300] = 0x7F80
    x[2, [300, 17]] = 0x7F80, 0xFF80
    x[3, 17] = 0x7FC0
    x[4, [0, k - 1]] = 0xFF80
    x[6, 64:72] = 0x7F80
    got = run(dev, x, d_w, n, k, len(blob))
    assert np.array_equal(got[[0, 5]], clean[[0, 5]])
    with np.errstate(invalid="ignore"):
        expect = np.stack([(O.bf16_to_f32(row).astype(np.float64) * dense).sum(axis=1) for row in x])
    special = [1, 2, 3, 4, 6]
    assert np.isinf(expect[special]).any() and np.isnan(expect[special]).any() and not np.isfinite(expect[special]).any()
    assert np.array_equal(O.bf16_to_f32(got[special]).astype(np.float64), expect[special], equal_nan=True)
    assert np.array_equal(run(dev, x[1:2], d_w, n, k, len(blob)), got[1:2])             # and alone
