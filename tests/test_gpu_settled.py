"""GPU tests of the shortcuts for activations that have settled: same bits as the oracle, which applies every layer."""
import numpy as np
import pytest

from conftest import rows_of
from graphchallenge21_b200 import SpDNN
from graphchallenge21_b200.generator import SyntheticNetwork, synthetic_images
from test_gpu_parity import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("env", [{}, {"SPDNN_FIXED_POINT": "0"}, {"SPDNN_WORD_RING": "7"}, {"SPDNN_BITS_SMALL": "1", "SPDNN_BITS_FIRST": "1"},
                                 {"SPDNN_STAGE_TABLES": "0"}],
                         ids=lambda e: ",".join(f"{k[6:]}={v}" for k, v in e.items()) or "default")
@pytest.mark.parametrize("n,b,lengths", [(1024, 200, range(81, 87)), (4096, 100, range(102, 110)), (16384, 40, (95, 103))])
def test_fixed_point_of_periodic_networks(n, b, lengths, env, monkeypatch, oracle):
    """The bit forms stop at the first period of the tables that maps a tile onto itself and apply only the layers
    behind the last whole period: network lengths of every remainder, images that are saturated from the start in
    patterns that move before they settle, images that die late."""
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    y0 = synthetic_images(n, b)
    y0[32:96] *= np.float32(32.0)
    y0[96:100] = np.float32(32.0)
    for L in lengths:
        net = SyntheticNetwork(n, L, "radix16")
        want = oracle.infer(y0, [(r, None) for r in rows_of(net)], float(net.bias), first_image=3)
        with SpDNN(n, L, float(net.bias)) as g:
            g.set_network(net)
            g.set_input_dense(y0, 3)
            res = g.infer()
            skipped = g.shortcuts()["skipped_layers"]
            check((g.categories().copy(), g.activations(), g.layer_live().copy(), res), want)
        assert 0 < len(want[0]) < b
        if "SPDNN_FIXED_POINT" in env:
            assert skipped == 0
        elif n == 1024 or "SPDNN_STAGE_TABLES" not in env:         # (a pre-pass that reads its tables from memory applies every layer)
            assert skipped > 0


@pytest.mark.parametrize("n,L,b,what,env,ends_early",
                         [(16384, 150, 40, "late", {}, True), (16384, 150, 40, "late", {"SPDNN_BITS_KERNEL": "0"}, True),
                          (16384, 150, 40, "blobs", {"SPDNN_BITS_KERNEL": "0"}, True), (65536, 80, 33, "late", {}, False),
                          (4096, 120, 70, "both", {"SPDNN_BITS_KERNEL": "0"}, True), (4096, 120, 70, "late", {"SPDNN_STAGE_TABLES": "0"}, True),
                          (1024, 120, 70, "both", {"SPDNN_TABLE_GROUP": "1"}, True), (1024, 120, 70, "both", {"SPDNN_TABLE_GROUP": "4"}, True),
                          (1024, 121, 70, "both", {"SPDNN_WORD_RING": "6"}, True), (1024, 121, 70, "both", {"SPDNN_WORD_RING": "5"}, False),
                          (1024, 122, 70, "blobs", {"SPDNN_TABLE_GROUP": "2", "SPDNN_WORD_RING": "9"}, True),
                          (1024, 123, 70, "both", {"SPDNN_FIXED_POINT": "0"}, False)])
def test_the_chunk_kernel_ends_at_a_fixed_point(n, L, b, what, env, ends_early, monkeypatch, oracle):
    """alt2_kernel's own bit form, without the pre-pass: images that saturate long after the last chunk began (bias 0 doubles
    a small value in every layer), table copies shorter than a period, word rings that just hold one or just do not."""
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    net = SyntheticNetwork(n, L, "radix16", bias=None if what == "blobs" else 0.0)
    y0 = synthetic_images(n, b)
    if what != "blobs":
        y0[slice(None) if what == "late" else slice(1, None, 2)] *= np.float32(2.0 ** -60)       # 32 in layer 65
    want_c, want_a, want_l = oracle.infer(y0, [(r, None) for r in rows_of(net)], float(net.bias))
    with SpDNN(n, L, float(net.bias)) as g:
        g.set_network(net)
        g.set_input_dense(y0)
        g.infer()
        skipped = g.shortcuts()["skipped_layers"]
        assert np.array_equal(g.layer_live(), want_l)
        assert np.array_equal(g.categories(), want_c)
        assert np.array_equal(g.activations(), want_a)
    assert len(want_c) > 0
    assert (skipped >= L - 100) if ends_early else skipped == 0, skipped
