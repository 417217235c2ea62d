"""GPU: calls from several threads."""

import threading

import pytest
import torch

from sage_b200 import SAGELinear, SPHQuantLinear, synthetic_sage, synthetic_sphquant

pytestmark = pytest.mark.gpu


def sage(k, n, seed, permuted=True):
    return SAGELinear({key: value.cuda() for key, value in synthetic_sage(k, n, seed=seed, permuted=permuted).items()}, n)


def sph(k, n, seed):
    return SPHQuantLinear({key: value.cuda() for key, value in synthetic_sphquant(k, n, seed=seed).items()})


def rows_of(m, k):
    return torch.randn(m, k, generator=torch.Generator().manual_seed(m)).half().cuda()


@pytest.mark.parametrize("make", [lambda: sage(1024, 256, 3, permuted=False), lambda: sph(1024, 256, 3)],
                         ids=["identity", "sphquant"])
def test_first_gpu_work_of_a_thread_is_a_tensor_map(make):
    """A call without a gather in front of the GEMM: the tensor map of its activations is made before anything else
    has given the thread a context."""
    layer, x = make(), rows_of(64, 1024)
    want, got = layer(x), []
    torch.cuda.synchronize()
    thread = threading.Thread(target=lambda: got.append(layer(x)))
    thread.start()
    thread.join()
    torch.cuda.synchronize()
    assert len(got) == 1 and torch.equal(want, got[0])
