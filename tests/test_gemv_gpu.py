"""GPU parity of the quantized GEMV against the CPU oracle, through the C ABI."""
import os

import numpy as np
import pytest
import torch

import oracle
from helpers import OP_RTOL, assert_close
from inferi_b200 import quant
from inferi_b200.ops import FfnGateUp, GemvQuant, GpuQuantTensor, InferiError, add_assign

pytestmark = pytest.mark.gpu
GOLDEN = np.load(os.path.join(os.path.dirname(__file__), "golden", "blocks.npz"))
QTYPES = [quant.Q8_0, quant.Q4_K, quant.Q5_K, quant.Q6_K]
LEGACY = [quant.Q4_0, quant.Q4_1, quant.Q5_0, quant.Q5_1]   # the reference's other GpuQuantTensor variants (op level, a kernel of their own)


def run_gemv(backend, qt, rows, cols, blocks, v):
    m = GpuQuantTensor(backend, qt, rows, cols, blocks)
    out = torch.full((rows,), float("nan"), device="cuda")
    GemvQuant.from_backend(backend).launch(out, m, torch.from_numpy(v).cuda())
    torch.cuda.synchronize()
    res = out.cpu().numpy()
    m.close()
    return res


@pytest.mark.parametrize("qt", QTYPES + LEGACY)
def test_golden_vectors(backend, qt):
    n = quant.NAMES[qt]
    rows, cols = GOLDEN[f"{n}_deq"].shape
    got = run_gemv(backend, qt, rows, cols, GOLDEN[f"{n}_blocks"], GOLDEN[f"{n}_v"])
    assert_close(got, GOLDEN[f"{n}_gemv"], what=f"golden {n}")


# shapes of the reference's own GEMV tests (crates/inferi/src/ops/gemv_quant.rs:502-816): 64 x 256, Q6_K 64 x 512,
# random scales with a quarter in the f16 subnormal range; plus aligned shapes that take the 128-bit kernels
@pytest.mark.parametrize("qt,rows,cols", [
    (quant.Q8_0, 64, 256), (quant.Q4_K, 64, 256), (quant.Q5_K, 64, 256), (quant.Q6_K, 64, 512),
    (quant.Q8_0, 64, 128), (quant.Q6_K, 8, 256), (quant.Q6_K, 64, 2048), (quant.Q6_K, 36, 6144), (quant.Q8_0, 260, 1024),
    (quant.Q4_K, 4, 256), (quant.Q4_K, 1000, 2560), (quant.Q4_K, 128, 11008), (quant.Q6_K, 64, 8192), (quant.Q8_0, 64, 14336),
    (quant.Q5_K, 296, 4096), (quant.Q4_K, 300, 6144), (quant.Q6_K, 1184, 4096), (quant.Q4_K, 2372, 2048), (quant.Q4_K, 16, 16384), (quant.Q4_K, 16, 16640), (quant.Q5_K, 12, 14336), (quant.Q4_K, 8, 32768), (quant.Q4_K, 8, 33024),
])
def test_reference_test_shapes_and_edges(backend, qt, rows, cols):
    _shape_case(backend, qt, rows, cols)


# the byte-balanced split of the rows over the pipelines (two per SM): fewer row pairs than pipelines, as many, one more, and a last
# range that ends inside a tile; rows of one block and of the streaming kernel's most
@pytest.mark.parametrize("rows", [4, 292, 588, 592, 596, 1180, 1188])
@pytest.mark.parametrize("qt,cols", [(quant.Q4_K, 256), (quant.Q5_K, 2048), (quant.Q8_0, 16384)])
def test_row_split(backend, qt, cols, rows):
    _shape_case(backend, qt, rows, cols)


# Rows so long that tiles hold 4 of them, two tiles at a time: CTAs with one tile, an odd and an even number of them, and none; the last warp of a row
# with one to four blocks
@pytest.mark.parametrize("rows", [4, 8, 588, 600, 1188, 1776, 1780, 2400, 4100])
@pytest.mark.parametrize("qt,cols", [(quant.Q4_K, 14336), (quant.Q4_K, 15104), (quant.Q5_K, 12800), (quant.Q6_K, 10240), (quant.Q8_0, 8704)])
def test_long_rows_two_tiles_at_a_time(backend, qt, cols, rows):
    _shape_case(backend, qt, rows, cols)


# the legacy formats at the shape of the reference's tests (gemv_quant.rs:502-816: 64 x 256; Q8_K blocks span 256 columns)
# and at a layer-sized one
@pytest.mark.parametrize("qt,rows,cols", [(q, 64, 256) for q in LEGACY + [quant.Q8_K]] + [(q, 512, 4096) for q in LEGACY + [quant.Q8_K]])
def test_legacy_formats(backend, qt, rows, cols):
    _shape_case(backend, qt, rows, cols)


# groups of 4 rows: one warp each, and 2, 4 or 8 warps that share the columns; rows of fewer blocks than a step, of whole steps and of a part more
# (their blocks then start at every multiple of 2 bytes); vectors off the 16-byte boundary
@pytest.mark.parametrize("qt", LEGACY)
@pytest.mark.parametrize("rows,cols", [(4, 32), (12, 96), (36, 224), (68, 4128), (2364, 288), (4740, 352), (9476, 64), (9480, 512)])
def test_legacy_splits(backend, qt, rows, cols):
    _shape_case(backend, qt, rows, cols)
    blocks = quant.random_blocks(qt, rows, cols, seed=rows)
    v = torch.randn(cols + 1, generator=torch.Generator().manual_seed(cols)).cuda()[1:]
    m = GpuQuantTensor(backend, qt, rows, cols, blocks)
    out = torch.full((rows,), float("nan"), device="cuda")
    GemvQuant(backend).launch(out, m, v)
    assert_close(out.cpu().numpy(), oracle.gemv_ref(qt, rows, cols, blocks, v.cpu().numpy()), what=f"{quant.NAMES[qt]} {rows}x{cols}")


# A power of two in front of the vector goes through to the result bit by bit (every operation is exact in it), up to elements or results near the
# largest float: no sum on the way exceeds it earlier.
@pytest.mark.parametrize("qt", LEGACY)
@pytest.mark.parametrize("rows,cols", [(12, 96), (9480, 512)])
def test_legacy_large_vectors(backend, qt, rows, cols):
    blocks = quant.random_blocks(qt, rows, cols, seed=rows)
    v = np.clip(np.random.default_rng(cols).standard_normal(cols), -4, 4).astype(np.float32)
    small = run_gemv(backend, qt, rows, cols, blocks, v)
    k = 126 - int(np.floor(np.log2(max(np.abs(small).max(), np.abs(v).max()))))   # the largest result or element is then at least 2^126
    big = run_gemv(backend, qt, rows, cols, blocks, np.ldexp(v, k))
    assert np.array_equal(big, np.ldexp(small, k))


# Q4_1, Q5_1: a weight is d q + m, and m is about -d times half of q's range.  Every weight is formed (rounded once, 2^-24) before it meets the vector; its
# products and their sums round as in the other formats: 1.0e-7 of the result's norm in all.  Adding up q's and the minimum's products apart,
# which nearly cancel, cost 3.4e-7 where the vector's mean is far from 0.
@pytest.mark.parametrize("qt", [quant.Q4_1, quant.Q5_1])
@pytest.mark.parametrize("mean", [0.0, 30.0])
def test_legacy_minimums_do_not_cost_accuracy(backend, qt, mean):
    rows, cols, five = 512, 4096, qt == quant.Q5_1
    rng = np.random.default_rng(qt)
    w = 0.02 * rng.standard_normal((rows, cols // 32, 32))
    d, m = ((w.max(-1) - w.min(-1)) / (31 if five else 15)).astype(np.float16), w.min(-1).astype(np.float16)
    q = np.clip(np.rint((w - m[..., None]) / d[..., None]), 0, 31 if five else 15).astype(np.uint8)
    parts = [d[..., None].view(np.uint8), m[..., None].view(np.uint8)]
    if five:
        parts.append(np.packbits(q >> 4, axis=-1, bitorder="little"))
    parts.append((q[..., :16] & 15) | ((q[..., 16:] & 15) << 4))
    blocks = np.concatenate(parts, -1).reshape(rows, -1)
    v = (rng.standard_normal(cols) + mean).astype(np.float32)
    want = (d.astype(np.float64)[..., None] * q + m.astype(np.float64)[..., None]).reshape(rows, cols) @ v.astype(np.float64)
    got = run_gemv(backend, qt, rows, cols, blocks, v)
    assert np.linalg.norm(got - want) <= 2e-7 * np.linalg.norm(want)


# A launch starts while the kernel before it still runs: the vector is read as that one leaves it, also where it was read before
@pytest.mark.parametrize("qt,rows,cols", [(quant.Q4_0, 512, 4096), (quant.Q5_1, 12464, 1024)])
def test_legacy_follows_the_kernel_that_writes_its_vector(backend, qt, rows, cols):
    m = GpuQuantTensor(backend, qt, rows, cols, quant.random_blocks(qt, rows, cols, seed=3))
    x, y = (torch.randn(cols, device="cuda", generator=torch.Generator(device="cuda").manual_seed(i)) for i in (1, 2))
    out, op = torch.zeros(60, rows, device="cuda"), GemvQuant(backend)
    z = x.clone()
    for i in range(60):
        add_assign(backend, x, y)
        op.launch(out[i], m, x)
    for i in range(60):
        z += y
        want = torch.zeros(rows, device="cuda")
        torch.cuda.synchronize()
        op.launch(want, m, z)
        torch.cuda.synchronize()
        assert torch.equal(out[i], want), i


def _shape_case(backend, qt, rows, cols):
    blocks = quant.random_blocks(qt, rows, cols, seed=rows * 31 + cols + qt, scale=1.0, subnormal_frac=0.25)
    v = np.random.default_rng(cols).standard_normal(cols).astype(np.float32)
    got = run_gemv(backend, qt, rows, cols, blocks, v)
    assert_close(got, oracle.gemv_ref(qt, rows, cols, blocks, v), what=f"{quant.NAMES[qt]} {rows}x{cols}")


@pytest.mark.parametrize("qt,rows,cols,seed", [
    (quant.Q8_0, 4096, 4096, 1001),      # single Q8_0 GEMV
    (quant.Q4_K, 4096, 4096, 2001), (quant.Q4_K, 14336, 4096, 2002), (quant.Q5_K, 4096, 14336, 2003),
    (quant.Q6_K, 128256, 4096, 2004),    # classifier
])
def test_benchmark_shapes(backend, qt, rows, cols, seed):
    blocks = quant.random_blocks(qt, rows, cols, seed=seed)
    v = np.random.default_rng(seed + 1).standard_normal(cols).astype(np.float32)
    got = run_gemv(backend, qt, rows, cols, blocks, v)
    ref = oracle.gemv_ref(qt, rows, cols, blocks, v)
    e = assert_close(got, ref, what=f"{quant.NAMES[qt]} {rows}x{cols}")
    assert e < 2e-4   # well inside the bar of 1e-3: the activations are 16-bit block fixed point (measured: 2e-5 .. 1.1e-4)
    # linearity in v (a size-independent property): W(2v) == 2 W v exactly in binary floating point
    got2 = run_gemv(backend, qt, rows, cols, blocks, 2 * v)
    assert np.array_equal(got2, 2 * got)


# where the streaming kernel's split changes: 1, 5, 9, 17, 32, 33 blocks of 256 columns (blocks per warp, warps per row, a last
# warp with fewer blocks), rows so long that it works on 4 instead of 8 of them (with 1, 2, 3 and 4 blocks in the last warp), and
# row counts that leave every SM a few rows more or less than whole tiles
@pytest.mark.parametrize("qt,rows,cols", [
    (quant.Q4_K, 1484, 256), (quant.Q4_K, 1484, 1280), (quant.Q5_K, 2372, 2304), (quant.Q8_0, 1484, 2304), (quant.Q5_K, 1484, 4352),
    (quant.Q4_K, 1484, 8192), (quant.Q6_K, 596, 8192), (quant.Q4_K, 1484, 8448), (quant.Q8_0, 1484, 8448), (quant.Q8_0, 300, 9728),
    (quant.Q8_0, 300, 9984), (quant.Q6_K, 1484, 10240), (quant.Q5_K, 300, 14336), (quant.Q4_K, 300, 16128),
])
def test_streaming_splits(backend, qt, rows, cols):
    _shape_case(backend, qt, rows, cols)
    # the fused gate/up launch: gate and up rows of a tile are worked on together
    g = quant.random_blocks(qt, rows, cols, seed=rows + cols)
    u = quant.random_blocks(qt, rows, cols, seed=rows + cols + 1)
    v = np.random.default_rng(cols + 1).standard_normal(cols).astype(np.float32)
    gm, um = (GpuQuantTensor(backend, qt, rows, cols, m) for m in (g, u))
    out = torch.empty(rows, device="cuda")
    FfnGateUp(backend).launch(out, gm, um, torch.from_numpy(v).cuda())
    a, b = (np.asarray(oracle.gemv_ref(qt, rows, cols, m, v), np.float64) for m in (g, u))
    # the product of two dot products, each within OP_RTOL
    assert_close(out.cpu().numpy(), b * a / (1 + np.exp(-np.maximum(a, -700.0))), rtol=2 * OP_RTOL, what=f"gate/up {quant.NAMES[qt]} {rows}x{cols}")


def test_f32_matrix_and_special_vectors(backend):
    rows, cols = 8, 300
    w = np.random.default_rng(1).standard_normal((rows, cols)).astype(np.float32)
    v = np.random.default_rng(2).standard_normal(cols).astype(np.float32)
    got = run_gemv(backend, quant.F32, rows, cols, w.view(np.uint8).reshape(rows, -1), v)
    assert_close(got, w.astype(np.float64) @ v, what="f32 gemv")
    # zero vector, and a vector with one huge entry per 32-group (dynamic range inside a group)
    blocks = quant.random_blocks(quant.Q4_K, 16, 1024, seed=5)
    assert np.array_equal(run_gemv(backend, quant.Q4_K, 16, 1024, blocks, np.zeros(1024, np.float32)), np.zeros(16, np.float32))
    v = np.random.default_rng(3).standard_normal(1024).astype(np.float32)
    v[::32] *= 1e4
    assert_close(run_gemv(backend, quant.Q4_K, 16, 1024, blocks, v), oracle.gemv_ref(quant.Q4_K, 16, 1024, blocks, v), what="wide range")


def test_host_buffer_entry_point(backend):
    blocks = quant.random_blocks(quant.Q6_K, 64, 2048, seed=9)
    v = np.random.default_rng(4).standard_normal(2048).astype(np.float32)
    m = GpuQuantTensor(backend, quant.Q6_K, 64, 2048, blocks)
    got = GemvQuant(backend).launch_host(m, v)
    assert_close(got, oracle.gemv_ref(quant.Q6_K, 64, 2048, blocks, v), what="host entry point")


def test_contract_violations_are_errors(backend):
    b = quant.random_blocks(quant.Q4_K, 8, 256, seed=1)
    with pytest.raises(InferiError):           # rows % 4 (the reference truncates silently)
        GpuQuantTensor(backend, quant.Q4_K, 6, 256, b[:6])
    with pytest.raises(InferiError):           # byte count
        GpuQuantTensor(backend, quant.Q4_K, 8, 512, b)
    with pytest.raises(InferiError):           # a GGUF type id this library has no reader for (Q2_K)
        GpuQuantTensor(backend, 10, 8, 256, b)
    m = GpuQuantTensor(backend, quant.Q4_K, 8, 256, b)
    with pytest.raises(InferiError):           # vector length
        GemvQuant(backend).launch(torch.zeros(8, device="cuda"), m, torch.zeros(128, device="cuda"))
    with pytest.raises(InferiError):           # host tensor where a device tensor is required
        GemvQuant(backend).launch(torch.zeros(8), m, torch.zeros(256, device="cuda"))


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("qt,rows,cols", [(quant.Q8_0, 64, 2048), (quant.Q4_K, 64, 2304), (quant.Q5_K, 64, 8448), (quant.Q6_K, 64, 2048), (quant.Q4_K, 8, 16640)])
def test_a_column_that_is_no_number_reaches_every_row(backend, qt, rows, cols, bad):
    """Every row of an f32 product with such a column is NaN or infinite; so is the fixed-point one (streaming kernel, and the
    wider rows' kernel).  The gate/up launch, which multiplies two such products, too."""
    blocks = quant.random_blocks(qt, rows, cols, seed=cols + qt)
    for at in (0, 37, cols - 1):
        v = np.random.default_rng(at).standard_normal(cols).astype(np.float32)
        v[at] = bad
        got = run_gemv(backend, qt, rows, cols, blocks, v)
        assert not np.isfinite(got).any()
        if np.isnan(bad):
            assert np.isnan(got).all()
    m = GpuQuantTensor(backend, qt, rows, cols, blocks)
    out = torch.zeros(rows, device="cuda")
    v[cols - 1] = float("nan")
    FfnGateUp(backend).launch(out, m, m, torch.from_numpy(v).cuda())
    assert torch.isnan(out).all()
    m.close()


@pytest.mark.parametrize("qt,rows,cols", [(quant.Q8_0, 64, 2048), (quant.Q4_K, 64, 2304), (quant.Q6_K, 64, 2048), (quant.Q4_K, 8, 16640)])
def test_views_off_the_vector_boundaries_are_refused(backend, qt, rows, cols):
    """The kernels read the input in 16-byte pieces and write pairs of rows: a contiguous view that starts in between is an error from the
    host, not a fault; one that starts on a boundary is taken."""
    blocks = quant.random_blocks(qt, rows, cols, seed=cols + qt)
    v = np.random.default_rng(qt).standard_normal(cols).astype(np.float32)
    ref = oracle.gemv_ref(qt, rows, cols, blocks, v)
    m = GpuQuantTensor(backend, qt, rows, cols, blocks)
    x, out = torch.zeros(cols + 4, device="cuda"), torch.zeros(rows + 2, device="cuda")
    wide = cols == 16640      # a row wider than the streaming kernel takes: its kernel writes single rows
    for at in (0, 1, 2, 3, 4):
        for to in (0, 1, 2):
            xv, ov = x[at:at + cols], out[to:to + rows]
            xv.copy_(torch.from_numpy(v))
            if at % 4 or (to % 2 and not wide):
                with pytest.raises(InferiError) as e:
                    GemvQuant(backend).launch(ov, m, xv)
                assert e.value.code == 1 and "aligned" in e.value.message
            else:
                GemvQuant(backend).launch(ov, m, xv)
                assert_close(ov.cpu().numpy(), ref, what=f"views at {at}, {to}")
    with pytest.raises(InferiError):
        FfnGateUp(backend).launch(out[:rows], m, m, x[:cols], norm_w=torch.ones(cols + 1, device="cuda")[1:])
    FfnGateUp(backend).launch(out[1:1 + rows], m, m, x[4:], norm_w=torch.ones(cols, device="cuda"))
    torch.cuda.synchronize()
    m.close()


@pytest.mark.parametrize("power", [-121, -115, -112, -100, 100, 108])
@pytest.mark.parametrize("qt,rows,cols", [(quant.Q8_0, 64, 2048), (quant.Q4_K, 64, 2304), (quant.Q5_K, 64, 8448), (quant.Q6_K, 64, 2048), (quant.Q4_K, 8, 16640)])
def test_vectors_far_from_one(backend, qt, rows, cols, power):
    """A vector times a power of two gives the product times it.  What is lost at the lower end is the group's scale, largest |x| / 32512,
    which f32 holds to a multiple of 2^-149: half of one of 2^(power + 1) / 32512 is 2^(-136 - power) of it, 3e-5 at 2^-121."""
    blocks = quant.random_blocks(qt, rows, cols, seed=cols + qt, scale=1e-3)
    v = np.clip(np.random.default_rng(power + 200).standard_normal(cols), -1.9, 1.9).astype(np.float32)
    got = np.ldexp(run_gemv(backend, qt, rows, cols, blocks, np.ldexp(v, power)).astype(np.float64), -power)
    assert_close(got, oracle.gemv_ref(qt, rows, cols, blocks, v), what=f"{quant.NAMES[qt]} {rows}x{cols} at 2^{power}")
