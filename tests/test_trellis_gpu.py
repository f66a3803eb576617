"""Trellis linear (prepass, tensor-core GEMM, epilogue, decode, scalar kernel) through the kernel-table ABI against
the oracle (modelled on native/tests/test_trellis.py)."""

import numpy as np
import pytest

from euhedral_b200 import layouts, sharding
from euhedral_b200.formats import LinearLaunch, TensorHandle, TrellisFormat, TrellisSettings
from euhedral_b200.gpu import KernelArguments
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


def random_object(rng, k, n, w, segments=1, scale=1.0):
    payload = rng.integers(-32768, 32768, size=(k // 16, n // 16, w), dtype=np.int16)
    suh = (rng.choice([-1.0, 1.0], size=(segments, k)) * rng.uniform(0.5, 2.0, size=(segments, k))).astype(np.float16)
    svh = (rng.uniform(0.01, 1.0, size=n) * scale).astype(np.float16)
    return payload, suh, svh


class DeviceLinear:
    def __init__(self, dev, payload, suh, svh, ends, target_ctas):
        self.dev = dev
        self.kt, self.nt, self.w = payload.shape
        self.k, self.n, self.ends = self.kt * 16, self.nt * 16, list(ends)
        layouts.trellis_validate_segments(self.ends, self.n)
        self.format = TrellisFormat(TrellisSettings(target_ctas=target_ctas))
        self.tensors = [dev.put(payload.astype("<i2")), dev.put(suh.astype("<f2")), dev.put(svh.astype("<f2")),
                        dev.put(np.array(self.ends, dtype="<i4"))]
        shapes = [payload.shape, (len(self.ends), self.k), (self.n,), (len(self.ends),)]
        self.handles = [TensorHandle(f"t{i}", tuple(shape), t.data_ptr(), t.numel()) for i, (t, shape) in enumerate(zip(self.tensors, shapes))]

    def linear(self, x_bits, row_exact=True, **select):
        rows = x_bits.shape[0]
        need = self.format.scratch_bytes(self.dev.gpu, rows, self.k, self.n, len(self.ends), row_exact=row_exact)
        d_x, d_y, d_s = self.dev.put(x_bits), self.dev.empty(rows * self.n * 2), self.dev.empty(need)
        launch = LinearLaunch(d_x.data_ptr(), d_y.data_ptr(), self.handles, rows, self.k, self.n, scratch=d_s.data_ptr(),
                              scratch_bytes=need, row_exact=row_exact)
        with self.dev.submit(**select) as gpu:
            self.format.linear(gpu, launch)
        return self.dev.get(d_y, np.uint16, (rows, self.n))

    def table_launches(self, x_bits, splits, **select):
        """The plan's launches through the kernel table, one by one: what every other way to a linear has to give, bit for bit."""
        rows, segments = x_bits.shape[0], len(self.ends)
        words, suh, svh, ends = [t.data_ptr() for t in self.tensors]
        d_x, d_act, d_y = self.dev.put(x_bits), self.dev.empty(segments * rows * self.k * 2), self.dev.empty(rows * self.n * 2)
        d_part = self.dev.empty(splits * rows * self.n * 4)
        with self.dev.submit(**select) as gpu:
            gpu.launch_table_kernel("TRELLIS_PREPASS", (self.k + 511) // 512, rows, segments, 128, 1, 1, 0,
                                    KernelArguments().pointer(d_x.data_ptr()).pointer(suh).pointer(d_act.data_ptr()).int32(rows).int32(self.k)
                                    .int32(segments).int32(0))
            gpu.launch_table_kernel("TRELLIS_MMA", self.n // 128, splits, 1, 256, 1, 1, 0,
                                    KernelArguments().pointer(d_act.data_ptr()).pointer(words).pointer(ends).pointer(svh).pointer(d_part.data_ptr())
                                    .pointer(d_y.data_ptr()).int32(rows).int32(self.k).int32(self.n).int32(self.w).int32(splits).int32(segments))
            if splits > 1:
                gpu.launch_table_kernel("TRELLIS_EPILOGUE", (self.n + 511) // 512, rows, 1, 128, 1, 1, 0,
                                        KernelArguments().pointer(d_part.data_ptr()).int32(splits).pointer(svh).pointer(d_y.data_ptr()).int32(rows)
                                        .int32(self.n))
        return self.dev.get(d_y, np.uint16, (rows, self.n))

    def own_count(self, x_bits, room=0, **select):
        """The linear with a split count of its own (splits = 0): (output, that count). Up to 8 rows it is read off the flags that the
        launch leaves, of more rows, in a scratch with room for the rotated activations, off the length of what is written."""
        rows, lib = x_bits.shape[0], self.dev.gpu.lib
        activations = layouts.align_up(len(self.ends) * rows * self.k * 2, 256) if rows > 8 and room else 0
        need = lib.euhedral_b200_linear_trellis_scratch_bytes(rows, self.k, self.n, len(self.ends), 0) + activations
        d_x, d_y, d_s = self.dev.put(x_bits), self.dev.empty(rows * self.n * 2), self.dev.empty(max(need, 256), fill=0xA5)
        with self.dev.submit(**select) as gpu:
            gpu.linear_trellis_bf16(d_x.data_ptr(), *[t.data_ptr() for t in self.tensors[:3]], self.tensors[3].data_ptr(), d_y.data_ptr(),
                                    d_s.data_ptr(), need, rows, self.k, self.n, self.w, len(self.ends), 0)
        left = self.dev.get(d_s, np.uint64, (max(need, 256) // 8,))
        count = 1
        if rows <= 8 and left[0] != 0xA5A5A5A5A5A5A5A5:
            blocks = self.n // 128
            joined = int(np.count_nonzero(left == left[0]))   # every block's flags end as one value
            assert joined % blocks == 0
            count = joined // blocks
        elif rows > 8:
            count = -(-(8 * int(np.flatnonzero(left != 0xA5A5A5A5A5A5A5A5)[-1]) + 8 - activations) // (rows * self.n * 4))
        return self.dev.get(d_y, np.uint16, (rows, self.n)), count

    def one_call(self, x_bits, splits, **select):
        """The same linear as one call (euhedral_b200_linear_trellis_bf16) with the split count given."""
        rows = x_bits.shape[0]
        need = self.dev.gpu.lib.euhedral_b200_linear_trellis_scratch_bytes(rows, self.k, self.n, len(self.ends), splits)
        d_x, d_y, d_s = self.dev.put(x_bits), self.dev.empty(rows * self.n * 2), self.dev.empty(max(need, 256), fill=0xA5)
        with self.dev.submit(**select) as gpu:
            gpu.linear_trellis_bf16(d_x.data_ptr(), *[t.data_ptr() for t in self.tensors[:3]], self.tensors[3].data_ptr(), d_y.data_ptr(),
                                    d_s.data_ptr(), need, rows, self.k, self.n, self.w, len(self.ends), splits)
        return self.dev.get(d_y, np.uint16, (rows, self.n))


def within_kernel_tolerance(got_bits, expect):
    """native/tests/test_trellis.py:157-165."""
    got = O.bf16_to_f32(got_bits).astype(np.float64)
    rms = float(np.sqrt(np.mean(expect ** 2)))
    return np.all(np.abs(got - expect) <= 0.004 * np.abs(expect) + 0.004 * rms)


@pytest.mark.parametrize("w", [16, 24, 32, 40, 48, 56, 64, 72, 80, 88, 96, 104, 112, 120, 128])
def test_decode_bf16_bitwise(dev, w):
    rng = np.random.default_rng(w)
    k, n = 128, 256
    payload, _, _ = random_object(rng, k, n, w)
    d_words, d_out = dev.put(payload.astype("<i2")), dev.empty(n * k * 2)
    with dev.submit() as gpu:
        gpu.launch_table_kernel("TRELLIS_DECODE_BF16", (k // 16) * (n // 16), 1, 1, 256, 1, 1, 0,
                                KernelArguments().pointer(d_words.data_ptr()).pointer(d_out.data_ptr()).int32(k).int32(n).int32(w))
    got = dev.get(d_out, np.uint16, (n, k))
    assert np.array_equal(got, O.bf16_bits(O.trellis_rotated_weight(payload).astype(np.float32).T))


@pytest.mark.parametrize("rows,k,s", [(3, 1024, 2), (203, 384, 3)])     # few rows: a warp per block; many: a thread per block
def test_prepass_bitwise(dev, rows, k, s):
    rng = np.random.default_rng(3)
    x = random_x(rng, rows, k)
    suh = (rng.choice([-1.0, 1.0], size=(s, k)) * rng.uniform(0.5, 2.0, size=(s, k))).astype(np.float16)
    d_x, d_suh, d_out = dev.put(x), dev.put(suh), dev.empty(s * rows * k * 2)
    for layout in (0, 1):
        with dev.submit() as gpu:
            gpu.launch_table_kernel("TRELLIS_PREPASS", (k + 511) // 512, rows, s, 128, 1, 1, 0,
                                    KernelArguments().pointer(d_x.data_ptr()).pointer(d_suh.data_ptr()).pointer(d_out.data_ptr())
                                    .int32(rows).int32(k).int32(s).int32(layout))
        got = dev.get(d_out, np.uint16, (s, rows, k))
        if layout == 0:
            expect = O.trellis_fragment_order(O.trellis_prepass(x, suh).view(np.uint16))
        else:
            rotated = O.hadamard128((O.bf16_to_f32(x)[None] * suh.astype(np.float32)[:, None, :]).astype(np.float32))
            expect = O.bf16_bits(rotated)
        assert np.array_equal(got, expect), layout


@pytest.mark.parametrize("w", [16, 24, 32, 40, 48, 56, 64, 72, 80, 88, 96, 104, 112, 120, 128])   # every stored width: every lane decoder
@pytest.mark.parametrize("target", [8, 140])
def test_tensor_core_route_matches_float64(dev, w, target):
    rng = np.random.default_rng(w + target)
    k, n = 1024, 512
    payload, suh, svh = random_object(rng, k, n, w, segments=2)
    linear = DeviceLinear(dev, payload, suh, svh, [256, 512], target)
    splits = TrellisFormat.splits(k, n, target)
    for rows in (1, 5, 8, 13, 40):
        x = random_x(rng, rows, k)
        expect = O.trellis_linear_f64(x, payload, suh, svh, [256, 512])
        got = linear.linear(x)
        assert within_kernel_tolerance(got, expect), (w, target, rows)
        if rows in (5, 13):
            assert np.array_equal(linear.one_call(x, splits), got), (w, target, rows)
            assert np.array_equal(linear.table_launches(x, splits), got), (w, target, rows)


# The layer's projection shapes (N x K) at the model's stored widths, one and two segments, through the operator's own
# launch plan for this device (K splits of 20, 20, 9 and 30 at 148 SMs: a split's tile rows are not a multiple of the 16
# the streaming stage holds, so stages reach past their split), against the plain-C restatement of the reference's
# linear (native/src/reference/trellis.cuh:14-55) within the reference's kernel tolerance.
@pytest.mark.parametrize("n,k", [(5120, 5120), (1024, 5120), (17408, 5120), (5120, 17408)])
@pytest.mark.parametrize("w", [40, 48, 56, 64])
def test_layer_shapes(dev, n, k, w):
    rng = np.random.default_rng(n + k + w)
    segments = 1 + (w // 8) % 2                       # 40, 56: two segments; 48, 64: one
    ends = [n] if segments == 1 else [n // 2, n]
    payload, suh, svh = random_object(rng, k, n, w, segments=segments)
    linear = DeviceLinear(dev, payload, suh, svh, ends, 8 * dev.gpu.multiprocessor_count())
    splits = TrellisFormat.splits(k, n, 8 * dev.gpu.multiprocessor_count())
    for rows in (1, 5):
        x = random_x(rng, rows, k)
        expect = OC.trellis_linear(x, payload, suh, svh, ends).astype(np.float64)
        got = linear.linear(x)
        assert within_kernel_tolerance(got, expect), (n, k, w, rows)
        assert np.array_equal(linear.one_call(x, splits, pdl=True), got), (n, k, w, rows)
        assert np.array_equal(linear.table_launches(x, splits, pdl=True), got), (n, k, w, rows)


def test_one_call_linear_is_bitwise_the_table_launches(dev):
    """The one-call linear and the operator's against the three table launches a host plans one by one."""
    rng = np.random.default_rng(44)
    k, n, w = 2048, 512, 48
    payload, suh, svh = random_object(rng, k, n, w, segments=2)
    ends = [256, 512]
    lib = dev.gpu.lib
    for target, rows in ((8, 3), (140, 5), (140, 1), (1, 7), (1, 20), (30, 13), (64, 40)):
        table = DeviceLinear(dev, payload, suh, svh, ends, target)
        x = random_x(rng, rows, k)
        splits = TrellisFormat.splits(k, n, target)
        expect = table.table_launches(x, splits)
        assert np.array_equal(table.linear(x), expect), (target, rows)
        assert np.array_equal(table.one_call(x, splits), expect), (target, rows)
        need = lib.euhedral_b200_linear_trellis_scratch_bytes(rows, k, n, 2, splits)
        # a flag per block and split, then the partials; nothing with one split
        assert need == (((n // 128 * splits * 8 + 255) & ~255) + splits * rows * n * 4 if splits > 1 else 0)
        d_x, d_y, d_s = dev.put(x), dev.empty(rows * n * 2), dev.empty(need)
        with dev.submit(pdl=True) as gpu:
            gpu.linear_trellis_bf16(d_x.data_ptr(), *[t.data_ptr() for t in table.tensors[:3]], table.tensors[3].data_ptr(), d_y.data_ptr(),
                                    d_s.data_ptr(), need, rows, k, n, w, 2, splits)
        assert np.array_equal(dev.get(d_y, np.uint16, (rows, n)), expect)
    # splits = 0 takes the device's default split count; a scratch that is too small is refused
    need = lib.euhedral_b200_linear_trellis_scratch_bytes(2, k, n, 2, 0)
    d_x, d_y, d_s = dev.put(random_x(rng, 2, k)), dev.empty(2 * n * 2), dev.empty(need)
    t = [h.data_ptr() for h in table.tensors]
    with dev.submit():
        assert lib.euhedral_b200_linear_trellis_bf16(d_x.data_ptr(), t[0], t[1], t[2], t[3], d_y.data_ptr(), d_s.data_ptr(), need, 2, k, n, w, 2, 0) == 0
        assert lib.euhedral_b200_linear_trellis_bf16(d_x.data_ptr(), t[0], t[1], t[2], t[3], d_y.data_ptr(), d_s.data_ptr(), 1024, 2, k, n, w, 2, 0) == -2


@pytest.mark.parametrize("k,n", [(16, 16), (48, 32), (80, 4112), (64, 16), (1040, 272), (4096, 2064)])
@pytest.mark.parametrize("w", [24, 64, 128])
def test_decode_bf16_of_odd_sizes(dev, w, k, n):
    """Fewer tiles along k than a warp takes at a time, a last unit that is not whole, more units than warps."""
    rng = np.random.default_rng(k * n + w)
    payload = rng.integers(0, 65536, (k // 16, n // 16, w), dtype=np.uint16)
    d_words, d_out = dev.put(payload.astype("<i2")), dev.put(np.full(n * k + 64, 0x1234, dtype=np.uint16))
    with dev.submit() as gpu:
        gpu.launch_table_kernel("TRELLIS_DECODE_BF16", (k // 16) * (n // 16), 1, 1, 256, 1, 1, 0,
                                KernelArguments().pointer(d_words.data_ptr()).pointer(d_out.data_ptr()).int32(k).int32(n).int32(w))
    got = dev.get(d_out, np.uint16, (n * k + 64,))
    assert np.array_equal(got[:n * k].reshape(n, k), O.bf16_bits(O.trellis_rotated_weight(payload).astype(np.float32).T))
    assert np.all(got[n * k:] == 0x1234)


@pytest.mark.parametrize("k,n,w,ends,target", [(2048, 512, 48, [256, 512], 140), (1408, 384, 64, [384], 64), (4224, 256, 56, [128, 256], 8), (1024, 640, 128, [640], 1)])
@pytest.mark.parametrize("rows", [1, 8, 9, 16, 17, 24, 25, 32, 33, 48, 49, 63])
def test_operator_is_bitwise_the_table_launches(dev, k, n, w, ends, target, rows):
    """What the operator queues as one call against the plan's launches through the kernel table, on both sides of every group of eight
    rows that a launch holds; in the operator's scratch and in one that has room for the partial sums only."""
    rng = np.random.default_rng(1000 * rows + k)
    payload, suh, svh = random_object(rng, k, n, w, segments=len(ends))
    linear = DeviceLinear(dev, payload, suh, svh, ends, target)
    x = random_x(rng, rows, k)
    splits = TrellisFormat.splits(k, n, target)
    expect = linear.table_launches(x, splits, pdl=True)
    words, d_suh, d_svh, d_ends = [t.data_ptr() for t in linear.tensors]
    d_x, d_part, d_y = dev.put(x), dev.empty(max(splits * rows * n * 4, 16)), dev.empty(rows * n * 2)
    assert np.array_equal(linear.linear(x), expect)
    with dev.submit(pdl=True) as gpu:
        gpu.linear_trellis_bf16(d_x.data_ptr(), words, d_suh, d_svh, d_ends, d_y.data_ptr(), d_part.data_ptr(), splits * rows * n * 4, rows, k, n, w,
                                len(ends), splits)
    assert np.array_equal(dev.get(d_y, np.uint16, (rows, n)), expect)


# The call that picks its split count itself (up to 8 rows one launch whose CTAs join the splits by flags) against the plan's launches at
# that count, on both sides of every group of eight rows, with and without room for the rotated activations. One and several segments,
# whole and half-step widths.
@pytest.mark.parametrize("k,n,w,ends", [(2048, 512, 48, [256, 512]), (1408, 384, 64, [384]), (4224, 256, 56, [128, 256]), (5120, 1024, 96, [1024])])
@pytest.mark.parametrize("rows", [1, 5, 8, 9, 16, 17, 24, 25, 32, 33, 40, 63, 97])
def test_own_split_count_is_bitwise_the_table_launches(dev, k, n, w, ends, rows):
    rng = np.random.default_rng(1000 * rows + k)
    payload, suh, svh = random_object(rng, k, n, w, segments=len(ends))
    linear = DeviceLinear(dev, payload, suh, svh, ends, 140)
    x = random_x(rng, rows, k)
    got, splits = linear.own_count(x, room=1, pdl=True)
    assert splits > 1
    assert np.array_equal(got, linear.table_launches(x, splits))
    again, _ = linear.own_count(x)
    assert np.array_equal(again, got)


def test_golden_linear_fixture(dev, golden):
    g = golden("trellis")
    linear = DeviceLinear(dev, g["linear_payload"], g["linear_suh"], g["linear_svh"], [256], 140)
    assert within_kernel_tolerance(linear.linear(g["linear_x"]), g["linear_y_f64"])
    two = DeviceLinear(dev, g["seg_payload"], g["seg_suh"], g["seg_svh"], list(g["seg_ends"]), 8)
    assert within_kernel_tolerance(two.linear(g["seg_x"]), g["seg_y_f64"])


def test_rows_are_bitwise_independent(dev):
    rng = np.random.default_rng(21)
    k, n, w = 1024, 256, 48
    payload, suh, svh = random_object(rng, k, n, w)
    for target in (2, 64):
        linear = DeviceLinear(dev, payload, suh, svh, [n], target)
        x = random_x(rng, 33, k)
        single = np.concatenate([linear.linear(x[r:r + 1]) for r in (0, 1, 7, 8, 32)])
        for rows in (2, 8, 9, 33):
            got = linear.linear(x[:rows])
            for at, r in enumerate((0, 1, 7, 8, 32)):
                if r < rows:
                    assert np.array_equal(got[r], single[at]), (target, rows, r)
        assert np.array_equal(linear.linear(x[:5], pdl=True), linear.linear(x[:5]))


# Verification of drafted tokens compares rows of a call of several with calls of one row: up to 63 rows, row-exact or not, a row has
# the same bits in the scratch that scratch_bytes names. Shapes with few and with many column blocks, whose K is cut often.
@pytest.mark.parametrize("n,k,segments", [(7168, 5120, 3), (14336, 2048, 1), (8320, 3072, 1), (5120, 8192, 3), (512, 1024, 2)])
def test_a_row_has_its_bits_in_every_call(dev, n, k, segments):
    rng = np.random.default_rng(n + k)
    ends = [n * (i + 1) // segments // 128 * 128 for i in range(segments)]
    payload, suh, svh = random_object(rng, k, n, 32, segments=segments)
    linear = DeviceLinear(dev, payload, suh, svh, ends, 8 * dev.gpu.multiprocessor_count())
    x = random_x(rng, 63, k)
    single = {r: linear.linear(x[r:r + 1], row_exact=False, pdl=True)[0] for r in (0, 1, 6, 14, 62)}
    for row_exact in (False, True):
        for rows in (1, 2, 7, 8, 9, 17, 63):
            got = linear.linear(x[:rows], row_exact=row_exact, pdl=True)
            for r, bits in single.items():
                assert r >= rows or np.array_equal(got[r], bits), (row_exact, rows, r)


def test_scalar_kernel_matches_float64(dev):
    rng = np.random.default_rng(22)
    k, n, w = 256, 256, 40
    payload, suh, svh = random_object(rng, k, n, w, segments=2)
    linear = DeviceLinear(dev, payload, suh, svh, [128, 256], 8)
    x = random_x(rng, 2, k)
    dev.gpu.select_exact_numerics(True)
    try:
        got = O.bf16_to_f32(linear.linear(x)).astype(np.float64)
    finally:
        dev.gpu.select_exact_numerics(False)
    expect = O.trellis_linear_f64(x, payload, suh, svh, [128, 256])
    assert np.all(np.abs(got - expect) <= np.abs(expect) * 2.0 ** -7 + np.max(np.abs(expect)) * 1e-3)


def test_column_shards_equal_the_whole(dev):
    """Cut at a segment boundary, with the K split fixed from the whole object's shape, a shard's columns are bitwise
    the whole object's."""
    rng = np.random.default_rng(23)
    k, n, w = 1024, 512, 48
    payload, suh, svh = random_object(rng, k, n, w, segments=2)
    ends = [256, 512]
    x = random_x(rng, 5, k)
    whole_splits = TrellisFormat.splits(k, n, 64)
    whole = DeviceLinear(dev, payload, suh, svh, ends, 64).linear(x)
    parts = []
    for first in (0, 256):
        p, s, v, e = sharding.trellis_rows(payload, suh, svh, ends, first, 256)
        # target chosen so that the shard's split count equals the whole object's
        shard = DeviceLinear(dev, p, s, v, e, whole_splits * (256 // 128))
        assert TrellisFormat.splits(k, 256, whole_splits * 2) == whole_splits
        parts.append(shard.linear(x))
    assert np.array_equal(np.concatenate(parts, axis=1), whole)


def test_table_abi(dev):
    lib = dev.gpu.lib
    names = [lib.euhedral_cuda_linear_kernel_name(i).decode() for i in range(lib.euhedral_cuda_linear_kernel_count())]
    assert names[:2] == ["euhedral_trellis_prepass", "euhedral_trellis_mma"] and names[4] == "euhedral_trellis_epilogue"
    assert dev.gpu.table_kernel_available("TRELLIS_MMA") and not dev.gpu.table_kernel_available("TRELLIS_MMA_ROWS_FP8")
    from euhedral_b200.gpu import GpuMemoryException
    with pytest.raises(GpuMemoryException) as wrong_count:
        dev.gpu.launch_table_kernel("TRELLIS_EPILOGUE", 1, 1, 1, 128, 1, 1, 0, KernelArguments().pointer(0).int32(1))
    assert wrong_count.value.status == -1
    with pytest.raises(GpuMemoryException) as wrong_width:
        dev.gpu.launch_table_kernel("TRELLIS_EPILOGUE", 1, 1, 1, 128, 1, 1, 0,
                                    KernelArguments().pointer(0).pointer(1).pointer(0).pointer(0).int32(1).int32(128))
    assert wrong_width.value.status == -1
    with pytest.raises(GpuMemoryException) as unavailable:
        dev.gpu.launch_table_kernel("TRELLIS_MMA_ROWS", 1, 1, 1, 256, 1, 1, 0, KernelArguments())
    assert unavailable.value.status == -5


@pytest.mark.parametrize("rows", [5, 20, 40])
@pytest.mark.parametrize("splits", [0, 9])
def test_one_call_linear_replayed_from_a_graph(dev, rows, splits):
    """A captured launch that joins its splits (splits = 0, up to 8 rows) carries the same flag tag on every replay: each replay must
    still wait for its own partial sums (the CTA that finishes a column block unsets the block's flags). More rows and a named count
    beside it."""
    torch = dev.torch
    rng = np.random.default_rng(45 + rows)
    k, n, w = 2048, 512, 48
    payload, suh, svh = random_object(rng, k, n, w)
    linear = DeviceLinear(dev, payload, suh, svh, [n], 140)
    lib = dev.gpu.lib
    need = lib.euhedral_b200_linear_trellis_scratch_bytes(rows, k, n, 1, splits)
    xs = [random_x(rng, rows, k) for _ in range(4)]
    count = splits or linear.own_count(xs[0], room=1)[1]
    assert count > 1
    d_x, d_y, d_s = dev.put(xs[0]), dev.empty(rows * n * 2), dev.empty(need)
    t = [h.data_ptr() for h in linear.tensors]
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream), dev.gpu.submit(stream.cuda_stream, pdl=True):
        args = (d_x.data_ptr(), t[0], t[1], t[2], t[3], d_y.data_ptr(), d_s.data_ptr(), need, rows, k, n, w, 1, splits)
        assert lib.euhedral_b200_linear_trellis_bf16(*args) == 0          # warm: plans and maps are made before the capture
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            assert lib.euhedral_b200_linear_trellis_bf16(*args) == 0
    for x in xs + xs[:1]:
        d_x.copy_(torch.from_numpy(x.view(np.uint8).reshape(-1).copy()))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        got = dev.get(d_y, np.uint16, (rows, n))
        d_y.fill_(0xA5)
        assert np.array_equal(got, linear.table_launches(x, count))


def test_one_launch_linear_replayed_from_a_graph(dev):
    """A captured linear with a named split count, replayed with changing inputs, against calls of its own."""
    torch = dev.torch
    rng = np.random.default_rng(45)
    k, n, w, rows = 2048, 512, 48, 5
    payload, suh, svh = random_object(rng, k, n, w)
    linear = DeviceLinear(dev, payload, suh, svh, [n], 140)
    splits = TrellisFormat.splits(k, n, 140)
    assert splits > 1
    lib = dev.gpu.lib
    need = lib.euhedral_b200_linear_trellis_scratch_bytes(rows, k, n, 1, splits)
    xs = [random_x(rng, rows, k) for _ in range(4)]
    d_x, d_y, d_s = dev.put(xs[0]), dev.empty(rows * n * 2), dev.empty(need)
    t = [h.data_ptr() for h in linear.tensors]
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream), dev.gpu.submit(stream.cuda_stream, pdl=True):
        args = (d_x.data_ptr(), t[0], t[1], t[2], t[3], d_y.data_ptr(), d_s.data_ptr(), need, rows, k, n, w, 1, splits)
        assert lib.euhedral_b200_linear_trellis_bf16(*args) == 0          # warm: plans and maps are made before the capture
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            assert lib.euhedral_b200_linear_trellis_bf16(*args) == 0
        for x in xs:
            d_x.copy_(torch.from_numpy(x.view(np.uint8).reshape(-1).copy()))
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert np.array_equal(dev.get(d_y, np.uint16, (rows, n)), linear.one_call(x, splits))
