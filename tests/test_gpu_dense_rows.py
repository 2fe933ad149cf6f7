"""The 4- and 8-row GEMV instances where their fixed-point sums are largest, and the memory of the
host-buffer call.

Constant rows make every quantised activation n = +-16256 and every group sum 32 (16) times that, the
largest its three byte planes hold; alternating signs make the sums vanish.  n * sx is then exact to
one rounding, so what is left against the f64 oracle is the f32 sum over the superblocks of numbers
up to S = sum |d sc q x| + |dmin m x|: (in_dim / 256 + 8) * 2^-24 * S."""
import threading

import numpy as np
import pytest
import torch

from cogni_ml_b200 import DeviceQuantWeight, QuantMatmul, QuantWeight, gemv_many, synth

pytestmark = pytest.mark.gpu
Q8_0, Q4_K, Q5_K, Q6_K, IQ4_NL = synth.Q8_0, synth.Q4_K, synth.Q5_K, synth.Q6_K, synth.IQ4_NL
TYPES = [Q8_0, Q4_K, Q5_K, Q6_K, IQ4_NL]


@pytest.mark.parametrize("qtype", TYPES)
@pytest.mark.parametrize("batch", [3, 4, 5, 6, 8])
@pytest.mark.parametrize("out_dim,in_dim", [(1, 256), (17, 2304), (48, 2048)])
def test_largest_group_sums(cuda, oracle, engine, qtype, batch, out_dim, in_dim):
    w = synth.make_weight(qtype, out_dim, in_dim, seed=61, tensor_id=qtype)
    x = np.ones((batch, in_dim), np.float32)
    x[1] = -3.0
    x[2, 1::2] = -1.0
    if batch > 4:
        x[4] = synth.make_activation(1, in_dim, seed=61)[0]
    dw = DeviceQuantWeight.upload(QuantWeight(w, qtype, out_dim, in_dim), cuda)
    y = dw.gemv(torch.from_numpy(x).to(cuda)).cpu().numpy()
    ref = oracle.matmul_add(x, batch, in_dim, w, qtype, out_dim, np.zeros(out_dim, np.float32)).reshape(batch, out_dim)
    deq = oracle.dequantize(qtype, w, out_dim * in_dim).reshape(out_dim, in_dim).astype(np.float64)
    # q * d and m * dmin are each at most twice the largest |weight| of a block plus the other: 4 covers both
    size = 4 * np.abs(x).astype(np.float64) @ np.abs(deq).T + 4 * np.abs(x).max(1)[:, None] * np.abs(deq).max(1)[None, :] * in_dim
    bound = (in_dim / 256 + 8) * 2.0 ** -24 * size
    if batch > 4:  # random row: activations in steps of 2^-14 of their superblock's largest
        bound[4] += 2.0 ** -14 * np.abs(x[4]).max() * np.abs(deq).sum(1)
    assert (np.abs(y - ref) <= bound).all()
    assert engine.lib.cogni_qmm_wait_timeouts() == 0


@pytest.mark.parametrize("qtype", TYPES)
@pytest.mark.parametrize("batch", [3, 4, 5, 8])
def test_fused_norm_of_one_superblock(cuda, oracle, qtype, batch):
    """The shortest rows: the norm's per-warp sums need more room than the rows' partial sums.  Activations
    are quantised in steps of 2^-14 of their superblock's largest, half a step each."""
    out_dim, in_dim = 100, 256
    w = synth.make_weight(qtype, out_dim, in_dim, seed=63, tensor_id=qtype)
    x = 3 * synth.make_activation(batch, in_dim, seed=63)
    wn = (1.0 + 0.1 * synth.make_activation(1, in_dim, seed=63, tensor_id=2)).ravel().astype(np.float32)
    dw = DeviceQuantWeight.upload(QuantWeight(w, qtype, out_dim, in_dim), cuda)
    y = gemv_many([dw], torch.from_numpy(x).to(cuda), norm_weight=torch.from_numpy(wn).to(cuda))[0].cpu().numpy()
    xn = oracle.rmsnorm(x, wn, 1e-6)
    ref = oracle.matmul_add(xn, batch, in_dim, w, qtype, out_dim, np.zeros(out_dim, np.float32)).reshape(batch, out_dim)
    deq = np.abs(oracle.dequantize(qtype, w, out_dim * in_dim).reshape(out_dim, in_dim).astype(np.float64))
    bound = 2.0 ** -14 * np.abs(xn).max(1)[:, None] * deq.sum(1)[None, :]
    assert (np.abs(y - ref) <= bound).all()


def test_host_calls_of_several_threads_and_sizes(cuda, oracle, engine):
    """Blocks are lent to one call at a time and reused by calls of other sizes; nothing of an earlier
    call shows; idle blocks go back on request and calls work after that."""
    cases = []
    for i, (qtype, out_dim, in_dim, rows) in enumerate([(Q4_K, 64, 512, 1), (Q8_0, 700, 2080, 3), (Q6_K, 16, 256, 2),
                                                        (IQ4_NL, 2000, 1024, 5), (Q5_K, 3000, 4096, 2)]):
        w = synth.make_weight(qtype, out_dim, in_dim, seed=71 + i, tensor_id=qtype)
        x = synth.make_activation(rows, in_dim, seed=71 + i)
        bias = np.linspace(-1, 1, out_dim, dtype=np.float32)
        ref = oracle.matmul_add(x, rows, in_dim, w, qtype, out_dim, bias)
        cases.append((x, rows, in_dim, w, qtype, out_dim, bias, np.asarray(ref).ravel()))
    failed = []

    def work(k):
        for c in (cases[k:] + cases[:k]) * 3:
            y = QuantMatmul.matmul_add(*c[:7])
            if not np.abs(y - c[7]).max() <= 1e-3 * np.abs(c[7]).max():
                failed.append((k, c[4]))

    for _ in range(2):
        threads = [threading.Thread(target=work, args=(k,)) for k in range(len(cases))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not failed
        assert engine.lib.cogni_qmm_release_host_workspaces() == 0
