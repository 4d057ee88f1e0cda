"""GPU parity of the tensor-core GEMM (the prefill building block) against the CPU oracle, through the C ABI.

`ib_gemm_quant` must give, for every input row, what the oracle's GEMV (dequantize + f64 dot) gives for that row."""
import numpy as np
import pytest
import torch

import oracle
from helpers import assert_close
from inferi_b200 import quant
from inferi_b200.ops import GemmQuant, GpuQuantTensor, InferiError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qt,rows,cols,n", [
    (quant.Q4_K, 128, 256, 16), (quant.Q4_K, 128, 256, 1), (quant.Q6_K, 128, 2048, 7), (quant.Q8_0, 256, 512, 33), (quant.Q5_K, 128, 1024, 128),
    (quant.Q4_K, 512, 2048, 32), (quant.Q6_K, 1024, 4096, 37), (quant.Q4_K, 4096, 4096, 128), (quant.Q4_K, 256, 14336, 5), (quant.Q6_K, 2048, 8192, 100),
    (quant.Q4_K, 384, 1024, 300),   # more rows than one pass takes: chunks of 128
    (quant.Q4_K, 14336, 4096, 96), (quant.Q5_K, 4096, 14336, 50),   # 1792 units over one wave of CTAs: tiles split between two or three of them
])
def test_gemm_matches_row_by_row_gemv(backend, qt, rows, cols, n):
    blocks = quant.random_blocks(qt, rows, cols, seed=rows + cols + n, scale=0.05)
    x = np.random.default_rng(n).standard_normal((n, cols)).astype(np.float32)
    m = GpuQuantTensor(backend, qt, rows, cols, blocks)
    out = torch.full((n, rows), float("nan"), device="cuda")
    GemmQuant(backend).launch(out, m, torch.from_numpy(x).cuda())
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    for t in sorted({0, n // 2, n - 1}):
        ref = oracle.gemv_ref(qt, rows, cols, blocks, x[t])
        e = assert_close(got[t], ref, what=f"gemm {quant.NAMES[qt]} {rows}x{cols} row {t} of {n}")
        assert e < 1e-4     # two f16 halves per split operand carry ~21 bits (the k-quant weights are exact integers)
    m.close()


@pytest.mark.parametrize("qt,rows,cols,n", [
    (quant.Q4_K, 128, 256, 129), (quant.Q5_K, 256, 512, 255), (quant.Q6_K, 128, 2048, 130), (quant.Q8_0, 384, 256, 257),   # edges of the 128-token chunks
    (quant.Q8_0, 128, 1024, 15), (quant.Q5_K, 128, 768, 17), (quant.Q6_K, 640, 4096, 1029),                                # ... of the 16-token padding, two passes
    (quant.Q4_K, 512, 14336, 130), (quant.Q5_K, 256, 2304, 1), (quant.Q8_0, 1024, 4096, 290), (quant.Q8_0, 1024, 4096, 300),   # dozens of planes, one column per thread; the result too large for that
])
def test_gemm_across_chunks_of_tokens(backend, qt, rows, cols, n):
    """Every row of the result: the tokens of all chunks, and the tiles whose K range is split between CTAs."""
    blocks = quant.random_blocks(qt, rows, cols, seed=rows + cols + n, scale=0.05)
    x = np.random.default_rng(n).standard_normal((n, cols)).astype(np.float32)
    m = GpuQuantTensor(backend, qt, rows, cols, blocks)
    out = torch.full((n, rows), float("nan"), device="cuda")
    GemmQuant(backend).launch(out, m, torch.from_numpy(x).cuda())
    w = torch.from_numpy(np.stack([oracle.dequantize(qt, blocks[r], cols) for r in range(rows)])).cuda().double()
    want = torch.from_numpy(x).cuda().double() @ w.T
    err = float((out.double() - want).norm() / want.norm())
    assert err < 1e-5      # operands carry >= 21 bits: 2^-21 per product, averaged over the sum
    assert float((out.double() - want).abs().max()) < 1e-4 * float(want.abs().max())
    m.close()


# from 512 tokens on several of them share a CTA of the kernel that splits the inputs: either side of the limit, rows of up to 4096 columns, of a few
# more, and of a part of the next 4096
@pytest.mark.parametrize("cols", [4096, 4352, 14336])
@pytest.mark.parametrize("n", [511, 513, 1030])
def test_gemm_inputs_of_many_tokens(backend, cols, n):
    test_gemm_across_chunks_of_tokens(backend, quant.Q4_K, 128, cols, n)


# a pair of SMs shares 256 rows and a chunk's tokens: an odd number of 128-row halves, halves with a remainder (up to 64 tokens such small matrices
# are one SM's work per tile)
@pytest.mark.parametrize("qt", [quant.Q4_K, quant.Q5_K, quant.Q6_K, quant.Q8_0])
@pytest.mark.parametrize("rows,n", [(128, 1), (384, 16), (384, 33), (640, 145)])
def test_gemm_halves_of_a_pair(backend, qt, rows, n):
    test_gemm_across_chunks_of_tokens(backend, qt, rows, 2048, n)


# 17 blocks per pair of SMs: the eight slots of the blocks' scales go round twice, and every block has scales of its own.  The same call gives the same bits.
@pytest.mark.parametrize("qt", [quant.Q4_K, quant.Q5_K, quant.Q6_K, quant.Q8_0])
def test_gemm_scales_of_long_ranges(backend, qt):
    rows, cols, n = 2048, 10240, 400
    test_gemm_across_chunks_of_tokens(backend, qt, rows, cols, n)
    m = GpuQuantTensor(backend, qt, rows, cols, quant.random_blocks(qt, rows, cols, seed=5, scale=0.05))
    x = torch.from_numpy(np.random.default_rng(6).standard_normal((n, cols)).astype(np.float32)).cuda()
    out = [torch.empty(n, rows, device="cuda") for _ in range(4)]
    for o in out:
        GemmQuant(backend).launch(o, m, x)
    assert all(torch.equal(o, out[0]) for o in out)
    m.close()


# one SM per tile up to 16 tokens, up to 64 where the matrix has no more 128 x 256 units than the GPU has SMs (148), a pair beyond: either side of each
# limit, and a last pass of a few tokens behind one of 1024
@pytest.mark.parametrize("qt", [quant.Q4_K, quant.Q5_K, quant.Q6_K, quant.Q8_0])
@pytest.mark.parametrize("rows,cols,n", [(128, 2048, 16), (2304, 2048, 64), (2304, 2048, 65), (2432, 2048, 16), (2432, 2048, 17), (384, 2048, 63), (256, 2048, 1030)])
def test_gemm_of_few_tokens(backend, qt, rows, cols, n):
    test_gemm_across_chunks_of_tokens(backend, qt, rows, cols, n)


@pytest.mark.parametrize("qt,rows,cols,n", [
    (quant.Q6_K, 128, 34816, 2), (quant.Q6_K, 256, 34816, 130), (quant.Q8_0, 128, 33024, 9),
])
def test_gemm_takes_rows_that_no_gemv_layout_holds(backend, qt, rows, cols, n):
    """Rows wider than the GEMV takes: twice, as the second call finds the first one's scratch, with another matrix in between."""
    x = torch.from_numpy(np.random.default_rng(n).standard_normal((n, cols)).astype(np.float32)).cuda()
    for seed in (1, 2, 1):
        blocks = quant.random_blocks(qt, rows, cols, seed=rows + cols + seed, scale=0.05)
        m = GpuQuantTensor(backend, qt, rows, cols, blocks)
        out = torch.full((n, rows), float("nan"), device="cuda")
        GemmQuant(backend).launch(out, m, x)
        w = torch.from_numpy(np.stack([oracle.dequantize(qt, blocks[r], cols) for r in range(rows)])).cuda().double()
        want = x.double() @ w.T
        assert float((out.double() - want).norm() / want.norm()) < 1e-5      # as above
        m.close()


@pytest.mark.parametrize("cols", [256, 768, 3072, 33024])
def test_gemm_rejects_rows_that_the_copies_cannot_take(backend, cols):
    m = GpuQuantTensor(backend, quant.Q6_K, 128, cols, quant.random_blocks(quant.Q6_K, 128, cols, seed=2))     # no multiple of 8 blocks
    with pytest.raises(InferiError) as e:
        GemmQuant(backend).launch(torch.empty(2, 128, device="cuda"), m, torch.zeros(2, cols, device="cuda"))
    assert e.value.code == 4
    m.close()


def test_gemm_rejects_shapes_outside_the_tensor_core_path(backend):
    blocks = quant.random_blocks(quant.Q4_K, 64, 256, seed=1)
    m = GpuQuantTensor(backend, quant.Q4_K, 64, 256, blocks)     # 64 rows: not a multiple of 128
    with pytest.raises(InferiError) as e:
        GemmQuant(backend).launch(torch.empty(2, 64, device="cuda"), m, torch.zeros(2, 256, device="cuda"))
    assert e.value.code == 4
    m.close()
