"""Sort_By_Key under a user comparator with values of user types: four bytes of alignment 1 and 2 beside
keys of 1 to 4 bytes (the value stage is filled by 4-byte asynchronous copies), and a type with member
initialisers, against a stable numpy sort."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def trtc(cuda):
    import thrustrtc_b200 as t
    t.init()
    t.Add_Code_Block("struct FourBytes { unsigned char b[4]; };\nstruct TwoHalves { short a = 1, b = 2; };\n"
                     "struct Small { unsigned char r, g; };\n")
    return t


@pytest.mark.parametrize("n", [300, 4097, 40_003])
@pytest.mark.parametrize("cls,size", [("FourBytes", 4), ("TwoHalves", 4), ("Small", 2)])
@pytest.mark.parametrize("kt,key_cls", [(np.int8, "int8_t"), (np.int16, "int16_t"), (np.int32, "int32_t")])
def test_values_of_user_types(trtc, n, cls, size, kt, key_cls):
    import torch
    rng = np.random.default_rng(n)
    k = rng.integers(-100, 101, n).astype(kt)
    v = rng.integers(0, 256, (n, size), dtype=np.uint8)
    tv = torch.from_numpy(v.copy()).cuda()
    dk = trtc.device_vector_from_numpy(k)
    comp = trtc.Functor({}, ["a", "b"], "        return (a < 0 ? -a : a) < (b < 0 ? -b : b);\n")
    trtc.Sort_By_Key(dk, trtc.DVVectorAdaptor(cls, n, tv.data_ptr(), tv), comp)
    order = np.argsort(np.abs(k.astype(np.int32)), kind="stable")
    assert dk.to_host().tobytes() == k[order].tobytes()
    assert tv.cpu().numpy().tobytes() == v[order].tobytes()
