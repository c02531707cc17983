"""The dispatches of the kernels at the sizes where they switch or leave a remainder, against the
CPU oracle (bit for bit where the results are integers or follow its rounding)."""
import numpy as np
import pytest

from rtlib_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _t(a, dev):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


@pytest.mark.parametrize("n", [1, 33, 227329, 909315])
def test_record_root_only(cuda, oracle, n):
    """A cleared tree sums its records in registers, four grid strides (227328 each) at a time."""
    from rtlib_b200.sdtree import SDTree
    rec = W.sdtree_records(n, n)
    rec["radiance"][::7] = np.nan
    wo = np.where(np.arange(n) % 5 == 0, 0.0, 2.0).astype(np.float32)
    sw = np.where(np.arange(n) % 11 == 0, -1.0, 0.5).astype(np.float32)
    delta = (np.arange(n) % 13 == 0).astype(np.uint8)
    g, o = SDTree((0, 0, 0), (1, 1, 1)), oracle.sdtree((0, 0, 0), (1, 1, 1))
    g.record(*(_t(rec[k], cuda) for k in ("pos", "uv", "radiance")), _t(wo, cuda), _t(sw, cuda), _t(delta, cuda))
    o.record(rec["pos"], rec["uv"], rec["radiance"], wo, sw, delta)
    eg, eo = g.export(sampling=False), o.export(sampling=False)
    np.testing.assert_array_equal(eg.scalars, eo.scalars)
    np.testing.assert_array_equal(eg.dsums, eo.dsums)


@pytest.mark.parametrize("threshold", [1 << 30, 4000, 300, 3])
def test_record_counter_placement(cuda, oracle, threshold):
    """One DTree of many quadrants (all counters in shared memory), tens and hundreds of DTrees
    (stat-weights only) and thousands (neither)."""
    from rtlib_b200.sdtree import SDTree
    rec = W.sdtree_records(1 << 15, 5)
    g, o = SDTree((0, 0, 0), (1, 1, 1)), oracle.sdtree((0, 0, 0), (1, 1, 1))
    args = [_t(rec[k], cuda) for k in ("pos", "uv", "radiance")]
    for _ in range(2):
        g.record(*args)
        o.record(rec["pos"], rec["uv"], rec["radiance"])
        g.build()
        o.build()
        g.refine(threshold)
        o.refine(threshold)
    g.record(*args)
    o.record(rec["pos"], rec["uv"], rec["radiance"])
    eg, eo = g.export(sampling=False), o.export(sampling=False)
    assert eg.topology == eo.topology
    np.testing.assert_array_equal(eg.scalars, eo.scalars)
    np.testing.assert_array_equal(eg.dsums, eo.dsums)
    assert g.status() == 0
