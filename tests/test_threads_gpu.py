"""GPU: calls from several threads."""

import threading

import pytest
import torch

from sage_b200 import SAGELinear, SPHQuantLinear, sage_grouped, synthetic_sage, synthetic_sphquant

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


class Grouped:
    """Two linears of one input in a grouped call, a staging and a decode launch."""

    def __init__(self, k, n, seed):
        self.packed, self.n = [list(synthetic_sage(k, n, seed=seed + i).values()) for i in range(2)], n
        self.packed = [[value.cuda() for value in values] for values in self.packed]

    def __call__(self, x):
        return torch.stack(sage_grouped([(x, *values) for values in self.packed], [self.n] * 2))


# calls of several launches through the scratch: gather and GEMM with and without K splits, staging and decode kernel
# with K slices, the second format's splits, grouped problems
CASES = {
    "gather_gemm": (sage, 2560, 1024, (33, 300, 64, 513)),
    "gather_split_gemm": (sage, 4096, 256, (48, 40, 130, 65)),
    "staging_sliced_decode": (sage, 9728, 512, (16, 9, 12, 8)),
    "sph_split_gemm": (sph, 4096, 256, (40, 64, 100, 33)),
    "grouped": (Grouped, 2560, 512, (16, 9, 12, 3)),
}


@pytest.mark.parametrize("name", CASES)
def test_threads_on_the_default_stream_do_not_share_scratch(name):
    make, k, n, rows = CASES[name]
    layers = [make(k, n, seed) for seed in range(len(rows))]
    inputs = [rows_of(m, k) for m in rows]
    alone = [layer(x) for layer, x in zip(layers, inputs)]
    torch.cuda.synchronize()
    outputs, errors = [[] for _ in rows], []
    start = threading.Barrier(len(rows))

    def work(i):
        try:
            start.wait()
            for _ in range(200):
                outputs[i].append(layers[i](inputs[i]))
        except Exception as error:  # noqa: BLE001 - reported by the test's own thread
            errors.append(error)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(rows))]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for want, got in zip(alone, outputs):  # (partial sums are added in a fixed order: the same bits)
        assert all(torch.equal(want, y) for y in got)
