"""Reduce_By_Key in its general form (segmented scan, then compaction of the segment tails) with outputs apart
from the inputs: elements above the one-pass form's 16 bytes of key and value, against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def t(cuda):
    import thrustrtc_b200 as m
    m.init()
    m.Add_Code_Block("struct Long2 { long long a, b; };\n")
    return m


@pytest.mark.parametrize("n", [1, 5000, 300_007])
def test_values_of_sixteen_bytes(t, n):
    import torch
    rng = np.random.default_rng(n)
    k = np.cumsum(rng.random(n) < 0.2).astype(np.int32)
    v = rng.integers(-1000, 1000, (n, 2))
    tv = torch.from_numpy(v.copy()).cuda()
    to = torch.zeros_like(tv)
    ko = t.device_vector_from_numpy(np.zeros(n, np.int32))
    op = t.Functor({}, ["x", "y"], "        auto r = x;\n        r.a += y.a;\n        r.b += y.b;\n        return r;\n")
    heads = np.flatnonzero(np.concatenate([[True], k[1:] != k[:-1]]))
    c = t.Reduce_By_Key(t.device_vector_from_numpy(k), t.DVVectorAdaptor("Long2", n, tv.data_ptr(), tv), ko,
                        t.DVVectorAdaptor("Long2", n, to.data_ptr(), to), t.EqualTo(), op)
    assert c == len(heads) and ko.to_host(0, c).tobytes() == k[heads].tobytes()
    assert to[:c].cpu().numpy().tobytes() == np.add.reduceat(v, heads, axis=0).tobytes()
