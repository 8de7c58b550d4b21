"""GPU tests of the launch schedule (SPDNN_PRINT_SCHEDULE): what a chunk may hold and which chunks get a pre-pass, each with
the results against the oracle."""
import re

import numpy as np
import pytest

from conftest import mixed_density_images
from graphchallenge21_b200 import SpDNN
from graphchallenge21_b200.generator import SyntheticNetwork, synthetic_images

pytestmark = pytest.mark.gpu


def schedule(capfd, monkeypatch, oracle, n, layers, bias, y0):
    """Runs the network, compares it with the oracle, returns the lines that were printed."""
    monkeypatch.setenv("SPDNN_PRINT_SCHEDULE", "1")
    want_c, want_a, want_l = oracle.infer(y0, layers, bias)
    capfd.readouterr()
    with SpDNN(n, len(layers), bias) as g:
        for l, (rows, vals) in enumerate(layers):
            g.set_layer_rows(l, rows, vals)
        g.set_input_dense(y0)
        g.infer()
        text = capfd.readouterr().err
        assert np.array_equal(g.layer_live(), want_l)
        assert np.array_equal(g.categories(), want_c)
        assert np.array_equal(g.activations(), want_a)
    return text.splitlines()


def chunks(lines, form):
    """(first, last) layer of the resident chunks of a form."""
    found = [re.search(r"resident layers (\d+)\.\.(\d+) .* (ALT2|GENERIC) ", line) for line in lines]
    return [(int(m[1]), int(m[2])) for m in found if m and m[3] == form]


def test_only_alt2_layers_take_the_rest_of_the_network_at_once(capfd, monkeypatch, oracle):
    """A network that stops being periodic inside its second chunk: the layers behind it have no tables that repeat."""
    n, first, L = 1024, 20, 240
    a, b = SyntheticNetwork(n, first, "radix16"), SyntheticNetwork(n, L - first, "random")
    layers = [(a.layer_rows(l) if l < first else b.layer_rows((l - first) % 6), None) for l in range(L)]
    y0 = np.concatenate([synthetic_images(n, 60), mixed_density_images(n, 60)])
    lines = schedule(capfd, monkeypatch, oracle, n, layers, float(a.bias), y0)
    assert chunks(lines, "ALT2") == [(1, 8), (9, 19)]
    assert chunks(lines, "GENERIC") == [(20, 147), (148, 239)]


@pytest.mark.parametrize("lengths,first", [("3,3,32", 7), ("1,1,1,60", 3), ("8,32", 41), ("20,20", None)])
def test_the_third_alt2_chunk_gets_the_pre_pass(lengths, first, capfd, monkeypatch, oracle):
    """... however short the first two are."""
    monkeypatch.setenv("SPDNN_CHUNKS", lengths)
    n, L = 4096, 60 if first else 40
    net = SyntheticNetwork(n, L, "radix16")
    y0 = synthetic_images(n, 70)
    y0[:32] *= np.float32(32.0)                                  # a tile that is saturated from the start
    lines = schedule(capfd, monkeypatch, oracle, n, [(net.layer_rows(l), None) for l in range(L)], float(net.bias), y0)
    found = [re.search(r"pre-pass for saturated tiles, layers (\d+)\.\.", line) for line in lines]
    starts = [int(m[1]) for m in found if m]
    assert starts[:1] == ([first] if first else [])
    assert starts == [c[0] for c in chunks(lines, "ALT2")][2:]
