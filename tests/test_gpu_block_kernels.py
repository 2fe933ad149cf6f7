"""Kernels that work block by block: the f32 GEMV of Q8_0 / IQ4_NL rows of any width and the
dequantiser's 16-byte stores, at the edges of their tiles, and their general forms for unaligned
buffers.

The GEMV computes d * q (exact quants, one rounding) and accumulates in f32: a lane adds at most 2
products in sequence per 256 columns and warp, the rest is a tree, so its error against the f64 oracle
stays below in_dim / 256 + 16 roundings of 2^-24 on the sum of the magnitudes; 1e-5 of max|y| has a
wide margin at these widths (measured 2e-7)."""
import numpy as np
import pytest
import torch

from cogni_ml_b200 import DeviceQuantWeight, QuantWeight, synth

pytestmark = pytest.mark.gpu
Q8_0, Q4_K, Q5_K, Q6_K, IQ4_NL = synth.Q8_0, synth.Q4_K, synth.Q5_K, synth.Q6_K, synth.IQ4_NL


def aligned_at(host: np.ndarray, offset: int, cuda) -> torch.Tensor:
    """`host` on the device, `offset` bytes past a 16-byte boundary."""
    raw = torch.from_numpy(np.ascontiguousarray(host).view(np.uint8).reshape(-1))
    buf = torch.empty(raw.numel() + 32, dtype=torch.uint8, device=cuda)
    start = (-buf.data_ptr()) % 16 + offset
    view = buf[start:start + raw.numel()]
    view.copy_(raw)
    return view


@pytest.mark.parametrize("qtype", [Q8_0, IQ4_NL])
@pytest.mark.parametrize("batch", [1, 2, 3, 4, 5, 6, 7, 9, 16, 19])
@pytest.mark.parametrize("out_dim,in_dim", [(1, 32), (37, 288), (1185, 2080), (2053, 2976), (4738, 544)])
def test_gemv_of_whole_blocks(cuda, oracle, qtype, batch, out_dim, in_dim):
    w = synth.make_weight(qtype, out_dim, in_dim, seed=41, tensor_id=qtype)
    x = synth.make_activation(batch, in_dim, seed=41)
    res = synth.make_activation(batch, out_dim, 41, 5)
    dw = DeviceQuantWeight.upload(QuantWeight(w, qtype, out_dim, in_dim), cuda)
    zero = np.zeros(out_dim, np.float32)
    ref = oracle.matmul_add(x, batch, in_dim, w, qtype, out_dim, zero, threads=oracle.max_threads()).reshape(batch, out_dim)
    y = torch.full((batch, out_dim), float("nan"), device=cuda)
    dw.gemv(torch.from_numpy(x).to(cuda), out=y, residual=torch.from_numpy(res).to(cuda))
    assert np.abs(y.cpu().numpy() - (ref + res)).max() <= 1e-5 * np.abs(ref).max()
    # activations on a 4-byte boundary take the row-per-warp kernel
    xo = aligned_at(x, 4, cuda).view(torch.float32).view(batch, in_dim)
    assert np.abs(dw.gemv(xo).cpu().numpy() - ref).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("qtype", [Q8_0, IQ4_NL])
@pytest.mark.parametrize("batch", [1, 2, 5])
def test_row_per_warp_kernel_on_request(cuda, oracle, engine, qtype, batch):
    """Kernel choice 1 runs the row-per-warp kernel: the bits of a call whose x no other kernel takes."""
    out_dim, in_dim = 301, 2976
    w = synth.make_weight(qtype, out_dim, in_dim, seed=49, tensor_id=qtype)
    x = synth.make_activation(batch, in_dim, seed=49)
    dw = DeviceQuantWeight.upload(QuantWeight(w, qtype, out_dim, in_dim), cuda)
    want = dw.gemv(aligned_at(x, 4, cuda).view(torch.float32).view(batch, in_dim))
    xd = torch.from_numpy(x).to(cuda)
    engine.lib.cogni_qmm_set_kernel_choice(1)
    try:
        assert torch.equal(dw.gemv(xd), want)
    finally:
        engine.lib.cogni_qmm_set_kernel_choice(0)
    assert not torch.equal(dw.gemv(xd), want)  # the block kernel adds in another order
    ref = oracle.matmul_add(x, batch, in_dim, w, qtype, out_dim, np.zeros(out_dim, np.float32)).reshape(batch, out_dim)
    assert np.abs(want.cpu().numpy() - ref).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("qtype,batch,out_dim,longest", [
    (Q8_0, 1, 37, 6), (IQ4_NL, 1, 5000, 6), (Q8_0, 2, 300, 3), (IQ4_NL, 2, 300, 6), (Q8_0, 4, 37, 3), (IQ4_NL, 7, 300, 1),
    (Q8_0, 9, 37, 0), (IQ4_NL, 1, 5001, 1), (Q8_0, 2, 5001, 1), (Q8_0, 3, 5001, 0)])
def test_short_rows_and_where_they_end(cuda, oracle, engine, qtype, batch, out_dim, longest):
    """Rows of up to `longest` blocks run on the row-per-warp kernel, the next longer ones do not; both
    against the oracle, with the tolerance of test_gemv_of_whole_blocks."""
    choose = engine.lib.cogni_qmm_set_kernel_choice
    for blocks in {1, longest, longest + 1} - {0}:
        in_dim = 32 * blocks
        w = synth.make_weight(qtype, out_dim, in_dim, seed=53, tensor_id=qtype)
        x = synth.make_activation(batch, in_dim, seed=53)
        dw = DeviceQuantWeight.upload(QuantWeight(w, qtype, out_dim, in_dim), cuda)
        xd = torch.from_numpy(x).to(cuda)
        y = dw.gemv(xd)
        choose(1)
        try:
            row_per_warp = torch.equal(y, dw.gemv(xd))
        finally:
            choose(0)
        assert row_per_warp == (blocks <= longest), f"{blocks} blocks"
        ref = oracle.matmul_add(x, batch, in_dim, w, qtype, out_dim, np.zeros(out_dim, np.float32)).reshape(batch, out_dim)
        assert np.abs(y.cpu().numpy() - ref).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("qtype,out_dim,in_dim,slabs", [
    (Q8_0, 700, 2976, 0), (IQ4_NL, 700, 2976, 0), (Q8_0, 9001, 288, 0), (IQ4_NL, 9001, 288, 0),  # block kernel
    (Q4_K, 700, 1024, 0), (IQ4_NL, 700, 1024, 0), (Q4_K, 597, 4096, 4), (Q6_K, 597, 12288, 3)])  # tiled, K slabs
def test_residual_in_place(cuda, engine, qtype, out_dim, in_dim, slabs):
    """The addend may be the output itself: the bits of a call with a separate residual, whatever the
    batch (groups of columns that do not divide it) and however often.  No oracle: both calls add the
    same sums."""
    w = synth.make_weight(qtype, out_dim, in_dim, seed=47, tensor_id=qtype)
    dw = DeviceQuantWeight.upload(QuantWeight(w, qtype, out_dim, in_dim), cuda)
    engine.lib.cogni_qmm_set_kernel_choice(60 + slabs)
    try:
        for batch in [*range(3, 17), 21]:
            x = torch.from_numpy(synth.make_activation(batch, in_dim, seed=47)).to(cuda)
            res = torch.from_numpy(synth.make_activation(batch, out_dim, 47, 5)).to(cuda)
            want = dw.gemv(x, residual=res)
            for _ in range(10):
                h = res.clone()
                dw.gemv(x, out=h, residual=h)
                assert torch.equal(h, want), f"batch {batch}: {int((h != want).sum())} values differ"
    finally:
        engine.lib.cogni_qmm_set_kernel_choice(60)


@pytest.mark.parametrize("qtype,elements", [(Q8_0, 1 << 18), (IQ4_NL, 3 << 16), (Q4_K, 3 << 19), (Q5_K, 3 << 20), (Q6_K, 3 << 20)])
@pytest.mark.parametrize("more", [-1, 0, 1, 33, 129])
@pytest.mark.parametrize("w_at,y_at", [(0, 0), (2, 0), (0, 4)])
def test_dequantize_from_where_the_wide_stores_begin(cuda, oracle, engine, qtype, elements, more, w_at, y_at):
    """The same at the sizes from which a tensor takes the 16-byte stores: whole CTAs of them, and remainders
    of one block and more."""
    n = elements + more * (32 if qtype in (Q8_0, IQ4_NL) else 256)
    w = synth.make_weight(qtype, 1, n, seed=45, tensor_id=qtype)
    raw = aligned_at(w, w_at, cuda)
    buf = torch.full((n + 8,), 7.0, device=cuda)
    start = (-buf.data_ptr()) % 16 // 4 + y_at // 4
    out = buf[start:start + n]
    st = engine.lib.cogni_qmm_dequantize(qtype, raw.data_ptr(), n, out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert st == 0
    assert np.array_equal(out.cpu().numpy().view(np.uint32), oracle.dequantize(qtype, w, n).view(np.uint32))
    assert buf[:start].eq(7.0).all() and buf[start + n:].eq(7.0).all()


@pytest.mark.parametrize("qtype", [Q8_0, Q4_K, Q5_K, Q6_K, IQ4_NL])
@pytest.mark.parametrize("blocks", [1, 7, 33, 129])
@pytest.mark.parametrize("w_at,y_at", [(0, 0), (2, 0), (0, 4)])
def test_dequantize_tiles_and_alignment(cuda, oracle, engine, qtype, blocks, w_at, y_at):
    be = 32 if qtype in (Q8_0, IQ4_NL) else 256
    n = blocks * be
    w = synth.make_weight(qtype, 1, n, seed=43, tensor_id=qtype)
    raw = aligned_at(w, w_at, cuda)
    buf = torch.full((n + 8,), 7.0, device=cuda)
    start = (-buf.data_ptr()) % 16 // 4 + y_at // 4
    out = buf[start:start + n]
    st = engine.lib.cogni_qmm_dequantize(qtype, raw.data_ptr(), n, out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert st == 0
    ref = oracle.dequantize(qtype, w, n)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), ref.view(np.uint32))
    assert buf[:start].eq(7.0).all() and buf[start + n:].eq(7.0).all()
