"""Reduce_By_Key of user value types of odd sizes beside small keys (results of 3 to 8 bytes in the pipeline's
ring), against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def trtc(cuda):
    import thrustrtc_b200 as t
    t.init()
    t.Add_Code_Block("\n".join("struct Bytes%d { unsigned char b[%d]; };" % (n, n) for n in (3, 5, 6, 7)) +
                     "\nstruct Halves3 { unsigned short b[3]; };\n")
    return t


@pytest.mark.parametrize("n", [5120, 50_011])
@pytest.mark.parametrize("kt", [np.int8, np.uint16])
@pytest.mark.parametrize("cls,count,dtype", [("Bytes3", 3, np.uint8), ("Bytes5", 5, np.uint8), ("Bytes6", 6, np.uint8),
                                             ("Bytes7", 7, np.uint8), ("Halves3", 3, np.uint16)])
def test_odd_value_types(trtc, n, kt, cls, count, dtype):
    import torch
    rng = np.random.default_rng(n + count)
    k = (np.cumsum(rng.random(n) < 0.1) % 100).astype(kt)
    v = rng.integers(0, 200, (n, count)).astype(dtype)
    tv = torch.from_numpy(v.view(np.uint8).copy()).cuda()
    to = torch.zeros_like(tv)
    ko = trtc.device_vector_from_numpy(np.zeros(n, kt))
    op = trtc.Functor({}, ["a", "b"], "        auto r = a;\n        for (int i = 0; i < %d; i++) if (b.b[i] > r.b[i]) r.b[i] = b.b[i];\n"
                                      "        return r;\n" % count)
    heads = np.flatnonzero(np.concatenate([[True], k[1:] != k[:-1]]))
    c = trtc.Reduce_By_Key(trtc.device_vector_from_numpy(k), trtc.DVVectorAdaptor(cls, n, tv.data_ptr(), tv), ko,
                           trtc.DVVectorAdaptor(cls, n, to.data_ptr(), to), trtc.EqualTo(), op)
    assert c == len(heads) and ko.to_host(0, c).tobytes() == k[heads].tobytes()
    assert to[:c].cpu().numpy().tobytes() == np.maximum.reduceat(v, heads, axis=0).tobytes()
