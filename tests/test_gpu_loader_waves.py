"""The device loader's waves at the edges of its passes and lanes: wave sizes
around a pass of the cluster's CTAs, fan-outs around the lanes that share an
element, one-element waves; equal to the host reader's netlist."""
import numpy as np
import pytest

from lsim_b200 import Simulator

pytestmark = pytest.mark.gpu


def _layers(widths, fan, seed):
    """A .ckt text: layer l has widths[l] gates, each reading one element of
    the layer before (element k feeds gates k * fan ... in turn) and one
    random earlier element; one PO per gate of the last layer."""
    rng = np.random.default_rng(seed)
    n_pi, n_po = widths[0], widths[-1]
    ids = [list(range(n_pi))]
    at = n_pi + n_po
    for w in widths[1:]:
        ids.append(list(range(at, at + w)))
        at += w
    sinks = {}
    for l in range(1, len(widths)):
        for k, g in enumerate(ids[l]):
            sinks.setdefault(ids[l - 1][(k // fan) % widths[l - 1]], []).append((g, 1))
            m = int(rng.integers(l))
            sinks.setdefault(ids[m][int(rng.integers(widths[m]))], []).append((g, 2))
    for k, g in enumerate(ids[-1]):
        sinks.setdefault(g, []).append((n_pi + k, 1))
    n_gates = sum(widths[1:])
    lines = ["%d\n%d\n%d\n%d" % (n_pi, n_po, n_gates, len(sinks))]
    lines += ["%d 0 %d %s" % (s, len(v), " ".join("%d %d" % p for p in v)) for s, v in sinks.items()]
    return "\n".join(lines) + "\n" + " ".join(str(int(t)) for t in rng.integers(1, 7, n_gates)) + "\n"


@pytest.mark.parametrize("widths,fan", [
    ([1, 1, 1, 1], 1), ([8, 255, 256, 257], 1), ([3, 2047, 2048, 2049, 5], 3), ([4100, 7, 4096], 64),
    ([5, 40, 300, 2400], 9), ([2, 8, 64, 512, 4096], 5)])
def test_waves_equal_the_host_reader(widths, fan):
    text = _layers(widths, fan, seed=sum(widths))
    dev, host = Simulator(0), Simulator(-1)
    dev.set_loader("device")
    dev.load_circuit(text)
    host.load_circuit(text)
    info = dev.load_info()
    assert info["on_device"] and not info["handed_back"]
    for f in ("gate_idx_to_tpg_order_idx", "levels", "types", "num_gates_per_level"):
        assert np.array_equal(getattr(dev, f)(), getattr(host, f)()), f
    assert dev.dot() == host.dot()
