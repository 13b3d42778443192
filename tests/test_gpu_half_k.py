"""Affines of long inner dimensions on a few hundred rows: two CTAs of a cluster take half of the inner dimension each."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# rows at the edges of the 64-row tiles and of the 32 rows a CTA keeps; ragged widths; odd numbers of 128-byte blocks and a last block that is not
# full; on 148 SMs the smallest (37) and largest (74) number of tiles and the first ones beyond (general plan)
@pytest.mark.parametrize("m,k,n", [(65, 2048, 2433), (96, 2048, 2500), (97, 2064, 2497), (128, 4096, 2560), (192, 2176, 1664), (500, 4000, 640), (2368, 2048, 128),
                                   (576, 4096, 1024), (2368, 2048, 256), (2369, 2048, 256), (512, 2048, 512), (2304, 2048, 128)])
@pytest.mark.parametrize("half,bias,relu", [(False, True, True), (True, True, False), (False, False, False)])
def test_half_of_k_per_cta(cuda_device, oracle, m, k, n, half, bias, relu):
    from marian_dev_b200 import ops
    rng = np.random.default_rng(m + k + n)
    a = rng.standard_normal((m, k)).astype(np.float32)
    w = (rng.standard_normal((k, n)) * 0.02).astype(np.float32)
    b = (rng.standard_normal(n) * 0.01).astype(np.float32) if bias else None
    bt, qb = oracle.prepare_b(w)
    want, want_acc, _aq, _qa = oracle.affine(a, bt, qb, b, 1.0, relu, want_acc=True)
    weight = ops.prepareB(torch.from_numpy(w).to(cuda_device))
    aq = ops.prepareA(torch.from_numpy(a).to(cuda_device))
    acc = torch.empty((m, n), dtype=torch.int32, device=cuda_device)
    bias_d = torch.from_numpy(b).to(cuda_device) if bias else None
    dtype = torch.float16 if half else torch.float32
    got = ops.multiply(aq, weight, bias_d, 1.0, relu, acc_out=acc, out_dtype=dtype)
    assert ops.poll_status() == 0
    assert np.array_equal(acc.cpu().numpy(), want_acc)
    assert np.array_equal(got.cpu().numpy(), want.astype(np.float16) if half else want)


# several matrices in one launch, each with a multiplier, a bias and an output of its own: 36 (general plan) to 74 tiles
@pytest.mark.parametrize("m,k,n_each,count", [(200, 2048, 384, 3), (250, 2048, 640, 2), (65, 4000, 1536, 3), (512, 2176, 384, 3), (130, 2064, 1024, 3)])
@pytest.mark.parametrize("half", [False, True])
def test_several_matrices(cuda_device, oracle, m, k, n_each, count, half):
    from tests.test_gpu_multi_weight import _run
    _run(cuda_device, oracle, m, k, n_each, count, with_bias=True, relu=half, out_dtype=torch.float16 if half else torch.float32)
