"""GPU tests of a context's life: what making, growing and ending one costs and what happens to a pass in flight meanwhile."""
import ctypes as C
import threading
import time

import numpy as np
import pytest

from conftest import mixed_density_images, rows_of
from graphchallenge21_b200 import SpDNN
from graphchallenge21_b200.generator import SyntheticNetwork, synthetic_images

pytestmark = pytest.mark.gpu


def fastest(f, times=8):
    best = float("inf")
    for _ in range(times):
        t = time.perf_counter()
        f()
        best = min(best, time.perf_counter() - t)
    return best


def test_a_new_context_costs_little_more_than_its_page_locked_block():
    """Making a context, giving it its first input and ending it, against the cost of page-locking a block and of asking
    for the device's properties (which nothing here needs as a whole) on the same machine."""
    import torch
    torch.zeros(1, device="cuda")
    rt = C.CDLL("libcudart.so.12")
    props = C.create_string_buffer(8192)

    def page_lock():
        p = C.c_void_p()
        assert rt.cudaMallocHost(C.byref(p), C.c_size_t(1 << 15)) == 0
        assert rt.cudaFreeHost(p) == 0

    y0 = synthetic_images(1024, 1)

    def life():
        with SpDNN(1024, 120, -0.3) as g:
            g.set_input_dense(y0)

    pinned, properties = fastest(page_lock), fastest(lambda: rt.cudaGetDeviceProperties_v2(props, 0))
    took = fastest(life)
    assert took < pinned + 0.5 * properties + 0.5e-3, (took, pinned, properties)


@pytest.mark.parametrize("pattern,n,L", [("random", 1024, 20), ("radix16", 1024, 60)])
def test_a_larger_input_while_a_pass_is_in_flight(pattern, n, L, oracle):
    """The buffers, device and page-locked, are replaced behind the pass, whose results are dropped."""
    net = SyntheticNetwork(n, L, pattern)
    images = mixed_density_images if pattern == "random" else synthetic_images
    sizes = (40, 700, 31, 3000, 3001, 64, 9000)
    y0 = images(n, max(sizes))
    with SpDNN(n, L, float(net.bias)) as g:
        g.set_network(net)
        for b in sizes:
            y = np.ascontiguousarray(y0[-b:])
            g.set_input_dense(y, b)
            g.infer_async()                      # the pass before is still running, or its results were never fetched
            if b in (700, 3001, 9000):
                want_c, want_a, want_l = oracle.infer(y, [(r, None) for r in rows_of(net)], float(net.bias), first_image=b)
                g.sync()
                assert np.array_equal(g.layer_live(), want_l)
                assert np.array_equal(g.categories(), want_c)
                assert np.array_equal(g.activations(), want_a)


def test_contexts_of_several_threads_come_and_go(oracle):
    n, L = 1024, 24
    net = SyntheticNetwork(n, L, "random")
    layers = [(r, None) for r in rows_of(net)]
    y0 = mixed_density_images(n, 2500)
    want = {b: oracle.infer(y0[:b], layers, float(net.bias)) for b in (1, 333, 2500)}
    wrong = []

    def work(seed):
        try:
            for it in range(6):
                b = (1, 333, 2500)[(seed + it) % 3]
                with SpDNN(n, L, float(net.bias)) as g:
                    g.set_network(net)
                    for bb in (b, 333):
                        g.set_input_dense(y0[:bb])
                        g.infer()
                        want_c, want_a, want_l = want[bb]
                        if not (np.array_equal(g.layer_live(), want_l) and np.array_equal(g.categories(), want_c)
                                and np.array_equal(g.activations(), want_a)):
                            wrong.append((seed, it, bb))
        except Exception as e:                   # noqa: BLE001 -- reported below
            wrong.append((seed, repr(e)))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
