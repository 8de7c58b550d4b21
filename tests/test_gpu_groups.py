"""GPU tests of the group sizes of GENERIC chunks: the batch, the classes and the entries of a layer decide how many images a
block holds (32 with one buffer and the outputs in registers, 16, 8 or 4 with two), every size against the oracle, bit for
bit."""
import numpy as np
import pytest

from conftest import mixed_density_images
from graphchallenge21_b200 import SpDNN
from graphchallenge21_b200.generator import SyntheticNetwork
from graphchallenge21_b200.network import pack_bits

pytestmark = pytest.mark.gpu


def network(n, L, k, seed):
    """Ragged columns (every tenth entry missing), every weight another value."""
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(L):
        rows = np.sort(np.argpartition(rng.random((n, n)), k, axis=1)[:, :k], axis=1).astype(np.int32)
        rows[rng.random(rows.shape) < 0.1] = -1
        out.append((rows, rng.uniform(0.02, 0.2, rows.shape).astype(np.float32)))
    return out


@pytest.mark.parametrize("batch", [4737, 2400, 1190, 70])
@pytest.mark.parametrize("n,k,L", [(96, 20, 11), (256, 37, 9), (512, 32, 9), (700, 9, 4), (1024, 32, 10)])
def test_general_weights(n, k, L, batch, oracle):
    layers = network(n, L, k, n + k)
    y0 = mixed_density_images(n, batch)
    y0[::5] *= np.float32(0.7)
    want_c, want_a, want_l = oracle.infer(y0, layers, -0.25, first_image=2)
    with SpDNN(n, L, -0.25) as g:
        for l, (rows, vals) in enumerate(layers):
            g.set_layer_rows(l, rows, vals)
        g.set_input_dense(y0, 2)
        res = g.infer()
        assert np.array_equal(g.layer_live(), want_l) and res.survivors == len(want_c)
        assert np.array_equal(g.categories(), want_c)
        assert np.array_equal(g.activations(), want_a)


@pytest.mark.parametrize("how", ["dense", "bits", "grey"])
@pytest.mark.parametrize("bias", [-0.3, 0.05])
@pytest.mark.parametrize("batch", [4737, 2400, 300])
def test_binary_words_are_read_in_place(batch, bias, how, oracle):
    n, L = 1024, 9
    net = SyntheticNetwork(n, L, "random", bias=bias)
    layers = [(net.layer_rows(l), None) for l in range(L)]
    y0 = mixed_density_images(n, batch)
    if how == "grey":
        y0[-1] *= np.float32(0.5)                    # one image that is not binary: all take the float tiles
    want_c, want_a, want_l = oracle.infer(y0, layers, bias)
    with SpDNN(n, L, bias) as g:
        g.set_network(net)
        for _ in range(2):
            if how == "bits":
                g.set_input_bits(pack_bits(y0))
            else:
                g.set_input_dense(y0)
            g.infer()
            assert np.array_equal(g.layer_live(), want_l)
            assert np.array_equal(g.categories(), want_c)
            assert np.array_equal(g.activations(), want_a)


@pytest.mark.parametrize("alternate", [False, True], ids=["one kind of layer", "a chunk per layer"])
def test_images_that_stay_unsaturated_keep_their_groups(alternate, oracle):
    """Every layer keeps the all-clip vector, but no image gets there: nothing is retired, and no chunk, however late, may
    be run in the small groups meant for the few images left behind retired ones."""
    n, L, k, b = 256, 60, 20, 2400
    rng = np.random.default_rng(3)
    layers = []
    for l in range(L):
        uniform = alternate and l % 2 == 1
        rows = np.sort(np.argpartition(rng.random((n, n)), k, axis=1)[:, :k], axis=1).astype(np.int32)
        if uniform:
            rows[:, 16:] = -1
        layers.append((rows, np.full((n, k), 1.0 / 16 if uniform else 1.002 / k, np.float32)))
    y0 = (8 + 8 * rng.random((b, n))).astype(np.float32)
    want_c, want_a, want_l = oracle.infer(y0, layers, 0.0)
    with SpDNN(n, L, 0.0) as g:
        for l, (rows, vals) in enumerate(layers):
            g.set_layer_rows(l, rows, vals)
        g.set_input_dense(y0)
        res = g.infer()
        assert np.array_equal(g.layer_live(), want_l) and len(want_c) == b
        assert np.array_equal(g.activations(), want_a) and ((want_a > 0) & (want_a < 32)).all()
        assert g.shortcuts()["retired_images"] == 0
        assert res.loop_launches == (L if alternate else 4)          # 8, 16, 32, 4 layers: the last has the small groups to choose from
        assert res.resident_group >= 16


def sm_count():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("n,k,L,uniform,per_sm,above,group",
                         [(96, 20, 5, False, 4, 0, 4), (96, 20, 5, False, 8, 1, 16), (96, 20, 5, False, 48, 1, 32),
                          (256, 37, 4, False, 4, 1, 8), (256, 37, 4, False, 48, 0, 16), (256, 37, 4, False, 48, 1, 32), (256, 32, 4, True, 8, 0, 8),
                          (512, 32, 4, False, 4, 0, 4), (512, 32, 4, False, 8, 0, 8), (512, 32, 4, False, 16, 0, 16), (512, 32, 4, False, 16, 1, 32),
                          (512, 32, 4, False, 32, 1, 32), (512, 32, 4, True, 8, 0, 8), (700, 9, 4, False, 4, 1, 8), (700, 9, 4, False, 16, 0, 16),
                          (700, 9, 4, False, 16, 1, 32), (700, 8, 4, False, 48, 1, 16), (1024, 32, 10, False, 4, 0, 4), (1024, 32, 10, False, 4, 1, 8),
                          (1024, 32, 10, False, 8, 1, 16), (1024, 32, 10, False, 16, 0, 16), (1024, 32, 10, False, 16, 1, 32),
                          (1024, 32, 4, True, 4, 0, 4), (1024, 32, 4, True, 8, 0, 4), (1024, 32, 4, True, 8, 1, 16), (1024, 20, 4, True, 8, 0, 8),
                          (1024, 32, 4, True, 16, 1, 32)])
def test_every_group_size_on_either_side_of_its_limits(n, k, L, uniform, per_sm, above, group, oracle):
    layers = network(n, L, k, n + k)
    if uniform:
        layers = [(rows, None) for rows, _ in layers]
    batch = per_sm * sm_count() + above              # the last batch of a class, or the first of the next
    y0 = mixed_density_images(n, batch)
    bias = -0.3 if uniform else -0.25
    want_c, want_a, want_l = oracle.infer(y0, layers, bias)
    with SpDNN(n, L, bias) as g:
        for l, (rows, vals) in enumerate(layers):
            g.set_layer_rows(l, rows, vals)
        g.set_input_dense(y0)
        res = g.infer()
        assert res.resident_group == group
        assert np.array_equal(g.layer_live(), want_l)
        assert np.array_equal(g.categories(), want_c)
        assert np.array_equal(g.activations(), want_a)


@pytest.mark.parametrize("n,k,big,small", [(256, 37, 6000, 64), (512, 20, 6000, 700), (1024, 32, 6000, 64), (1024, 4, 5000, 900)])
def test_a_small_batch_runs_alike_whatever_the_context_has_served(n, k, big, small, oracle):
    """The plan follows the batch, not the buffers: sizes in turn through one context, each as in a context of its own."""
    L = 5
    layers = network(n, L, k, n + k)
    y0 = mixed_density_images(n, big)

    def context():
        g = SpDNN(n, L, -0.25)
        for l, (rows, vals) in enumerate(layers):
            g.set_layer_rows(l, rows, vals)
        return g

    with context() as used:
        for b in (big, small, big, 1, small):
            y = y0[:b] * np.float32(0.9 if b == small else 1.0)
            want_c, want_a, want_l = oracle.infer(y, layers, -0.25)
            used.set_input_dense(y)
            res = used.infer()
            with context() as fresh:
                fresh.set_input_dense(y)
                own = fresh.infer()
            assert (res.resident_group, res.loop_launches) == (own.resident_group, own.loop_launches)
            assert np.array_equal(used.layer_live(), want_l)
            assert np.array_equal(used.categories(), want_c)
            assert np.array_equal(used.activations(), want_a)


def test_only_full_batches_split_their_first_chunk(oracle):
    n, L = 16384, 24
    net = SyntheticNetwork(n, L, "radix16")
    big = 128 * sm_count() + 1
    rng = np.random.default_rng(1)
    bits = rng.integers(0, 256, (big, n // 8), dtype=np.uint8)
    y0 = mixed_density_images(n, 40)
    want_c, want_a, want_l = oracle.infer(y0, [(net.layer_rows(l), None) for l in range(L)], float(net.bias))
    with SpDNN(n, L, float(net.bias)) as g:
        g.set_network(net)
        g.set_input_dense(y0)
        fresh = g.infer().loop_launches
        g.set_input_bits(bits)
        assert g.infer().loop_launches == fresh + 1
        g.set_input_bits(bits[:-1])
        assert g.infer().loop_launches == fresh
        g.set_input_dense(y0)
        assert g.infer().loop_launches == fresh
        assert np.array_equal(g.layer_live(), want_l)
        assert np.array_equal(g.categories(), want_c)
        assert np.array_equal(g.activations(), want_a)


@pytest.mark.parametrize("k,per_sm,launches", [(4, 30, 4), (20, 30, 4), (4, 50, 4), (12, 50, 7), (20, 50, 7)])
def test_only_large_batches_of_long_columns_get_short_chunks(k, per_sm, launches, oracle):
    """Weights that keep the all-clip vector, images of which some get there and some stay unsaturated."""
    n, L, b = 96, 60, per_sm * sm_count() + 5
    rng = np.random.default_rng(k)
    rows = [np.sort(np.argpartition(rng.random((n, n)), k, axis=1)[:, :k], axis=1).astype(np.int32) for _ in range(3)]
    layers = [(rows[l % 3], np.full((n, k), 1.002 / k, np.float32)) for l in range(L)]
    y0 = (8 + 8 * rng.random((b, n))).astype(np.float32)
    y0[::3] = 31.5 + 0.5 * rng.random((len(y0[::3]), n))
    want_c, want_a, want_l = oracle.infer(y0, layers, 0.0)
    with SpDNN(n, L, 0.0) as g:
        for l, (r, v) in enumerate(layers):
            g.set_layer_rows(l, r, v)
        g.set_input_dense(y0)
        res = g.infer()
        assert res.loop_launches == launches                     # 8, 16, 32, 4 or 8, 2, 2, 4, 8, 16, 20 layers
        assert np.array_equal(g.layer_live(), want_l)
        assert np.array_equal(g.categories(), want_c)
        assert np.array_equal(g.activations(), want_a)
        retired = g.shortcuts()["retired_images"]
    top = (want_a == 32).all(axis=1).sum()
    assert 0 < retired <= top < b
