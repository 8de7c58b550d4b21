"""GPU tests of retired images (every activation clip, every later layer keeps that): same bits as the oracle, which
applies every layer to every image."""
import numpy as np
import pytest

from conftest import mixed_density_images, rows_of
from graphchallenge21_b200 import SpDNN
from graphchallenge21_b200.generator import SyntheticNetwork, synthetic_images

pytestmark = pytest.mark.gpu


def run(n, layers, bias, clip, y0, first):
    with SpDNN(n, len(layers), bias, clip=clip) as g:
        for l, (rows, vals) in enumerate(layers):
            g.set_layer_rows(l, rows, vals)
        out = []
        for part in (y0, y0[: max(1, len(y0) // 3)]):          # a second, smaller batch in the same buffers
            g.set_input_dense(part, first)
            res = g.infer()
            out.append((g.categories().copy(), g.activations(), g.layer_live().copy(), res.survivors, g.shortcuts()["retired_images"]))
        return out


@pytest.mark.parametrize("env", [{}, {"SPDNN_RETIRE": "0"}, {"SPDNN_RESIDENT": "0"}, {"SPDNN_CHUNK_FIRST": "3"}, {"SPDNN_BITS_FIRST": "1"},
                                 {"SPDNN_STAGE_TABLES": "0"}],
                         ids=lambda e: ",".join(f"{k[6:]}={v}" for k, v in e.items()) or "default")
@pytest.mark.parametrize("kind,n,b,L", [("random", 1024, 333, 26), ("random", 1024, 64, 9), ("random", 16384, 37, 18), ("radix16", 1024, 200, 61),
                                        ("radix16", 4096, 97, 60), ("radix16", 16384, 65, 50), ("hole", 1024, 200, 24), ("general", 512, 150, 14),
                                        ("all", 1024, 40, 12)])
def test_retired_images_are_survivors(kind, n, b, L, env, monkeypatch, oracle):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    net = SyntheticNetwork(n, L, "radix16" if kind == "radix16" else "random")
    bias, clip = float(net.bias), 32.0
    layers = [(r, None) for r in rows_of(net)]
    y0 = synthetic_images(n, b) if kind == "radix16" else mixed_density_images(n, b)
    if kind == "hole":                       # one layer in mid-network does not keep the all-clip vector
        rows = layers[13][0].copy()
        rows[5] = -1
        layers[13] = (rows, None)
    if kind == "general":
        rng = np.random.default_rng(7)
        layers = [(r, rng.uniform(0.02, 0.2, r.shape).astype(np.float32)) for r, _ in layers]
        bias = -0.25
    if kind == "all":                        # every image at clip from the start, next to dead ones
        y0[:] = clip
        y0[::7] = 0.0
    got = run(n, layers, bias, clip, y0, 11)
    for part, (cats, act, live, survivors, retired) in zip((y0, y0[: max(1, b // 3)]), got):
        wc, wa, wl = oracle.infer(part, layers, bias, clip=clip, first_image=11)
        assert np.array_equal(live, wl)
        assert np.array_equal(cats, wc) and survivors == len(wc)
        assert np.array_equal(act, wa)
        assert retired <= (wa == clip).all(axis=1).sum()
        if "SPDNN_RETIRE" in env:
            assert retired == 0
        elif n < 16384 and L >= 12 and kind in ("random", "general", "all"):
            assert retired > 0


def test_large_batches_retire_in_short_chunks(oracle):
    import torch
    n, L, b = 1024, 26, 48 * torch.cuda.get_device_properties(0).multi_processor_count + 37
    net = SyntheticNetwork(n, L, "random")
    y0 = mixed_density_images(n, b)
    want_c, want_a, want_l = oracle.infer(y0, [(r, None) for r in rows_of(net)], float(net.bias), first_image=11)
    with SpDNN(n, L, float(net.bias)) as g:
        g.set_network(net)
        g.set_input_dense(y0, 11)
        res = g.infer()
        assert res.loop_launches == 6                            # 8, 2, 2, 4, 8, 2 layers
        assert g.shortcuts()["retired_images"] > 0.4 * b
        assert np.array_equal(g.layer_live(), want_l)
        assert np.array_equal(g.categories(), want_c)
        assert np.array_equal(g.activations(), want_a)


def _column_value(clip, weights, bias, uniform):
    """What a column of an all-clip input yields before it is cut off at clip, rounded step by step as the kernels do."""
    s = np.float32(0)
    for w in weights:
        s = np.float32(s + (clip if uniform else np.float32(clip * w)))
    if uniform:
        s = np.float32(s * weights[0])
    return np.float32(s + bias)


@pytest.mark.parametrize("clip", [32.0, 2.5, 0.1])
@pytest.mark.parametrize("kind", ["general", "uniform", "short", "empty"])
def test_the_last_bit_decides_whether_a_layer_keeps_the_top(kind, clip, oracle):
    """One column of one layer yields clip, or the number below it: all images are all clip until then."""
    n, L, k, b = 64, 14, 16, 50
    rng = np.random.default_rng(11)
    clip = np.float32(clip)
    rows = [np.sort(np.argpartition(rng.random((n, n)), k, axis=1)[:, :k], axis=1).astype(np.int32) for _ in range(L)]
    vals = [rng.uniform(0.1, 0.2, (n, k)).astype(np.float32) for _ in range(L)]
    uniform = kind != "general"
    variants = []
    if kind == "general":
        bias = np.float32(-0.1 * clip)
        w = vals[11][5]
        w[:] = np.float32(0.06)                            # too little without the last one; the least last one that does
        lo, hi = np.float32(0.0), np.float32(1.0)
        while np.nextafter(lo, hi) < hi:
            mid = np.float32((lo + hi) / 2)
            if mid in (lo, hi):
                break
            w[-1] = mid
            lo, hi = (lo, mid) if _column_value(clip, w, bias, False) >= clip else (mid, hi)
        for last, keeps in ((hi, True), (lo, False)):
            v = [x.copy() for x in vals]
            v[11][5, -1] = last
            assert (_column_value(clip, v[11][5], bias, False) >= clip) == keeps
            variants.append((rows, v, bias, keeps))
    else:
        vals = [np.full((n, k), 0.0625, np.float32) for _ in range(L)]
        below = np.float32(clip - np.nextafter(clip, np.float32(0)))
        if kind == "uniform":                              # 16 times clip / 16, and too little bias to matter or enough
            biases = [np.float32(f * below) for f in (0.0, -0.25, -0.75, -1.0, -3.0, -9.0)]
            variants = [(rows, vals, x, bool(_column_value(clip, vals[0][0], x, True) >= clip)) for x in biases]
            assert variants[0][3] and not variants[-1][3]
        else:
            short = [r.copy() for r in rows]
            short[11][5, 15 if kind == "short" else 0:] = -1
            variants = [(short, vals, np.float32(0), False), (rows, vals, np.float32(0), True)]
    y0 = np.full((b, n), clip, np.float32)
    for r, v, bias, keeps in variants:
        layers = [(x, None if uniform else y) for x, y in zip(r, v)]
        want_c, want_a, want_l = oracle.infer(y0, layers, float(bias), clip=float(clip))
        with SpDNN(n, L, float(bias), clip=float(clip)) as g:
            for l, (x, y) in enumerate(layers):
                g.set_layer_rows(l, x, y)
            g.set_input_dense(y0)
            g.infer()
            assert np.array_equal(g.layer_live(), want_l)
            assert np.array_equal(g.categories(), want_c)
            assert np.array_equal(g.activations(), want_a)
            assert g.shortcuts()["retired_images"] == (b if keeps else 0)
