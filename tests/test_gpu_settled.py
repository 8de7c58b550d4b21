"""GPU tests of the shortcuts for activations that have settled: same bits as the oracle, which applies every layer."""
import numpy as np
import pytest

from conftest import rows_of
from graphchallenge21_b200.generator import SyntheticNetwork, synthetic_images
from test_gpu_parity import check, run_gpu

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
        check(run_gpu(net, y0, first=3, alias=True), want)
        assert 0 < len(want[0]) < b
