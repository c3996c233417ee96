"""A tuning table belongs to the kernels it was measured with: one of an earlier
version is neither loaded from a cache file nor accepted by hand.  No GPU."""
import ctypes

from nbodyssey_b200 import _lib as L

# the tables measured before the all-pairs, sort and build kernels of version 3
EARLIER = 2


def _table(version):
    t = L.nb_tune_table()
    L.check(L.load().nb_tune_defaults(ctypes.byref(t)))
    t.version = version
    return t


def test_a_cache_of_earlier_kernels_is_not_loaded(tmp_path):
    lib = L.load()
    path = tmp_path / "tune.bin"
    path.write_bytes(bytes(_table(EARLIER)))
    assert lib.nb_tune_load(str(path).encode()) == L.NB_ERR_NOTFOUND
    assert lib.nb_tune_set(ctypes.byref(_table(EARLIER))) == L.NB_ERR_INVALID


def test_the_binding_and_the_library_agree():
    t = L.nb_tune_table()
    L.check(L.load().nb_tune_defaults(ctypes.byref(t)))
    assert t.version == L.NB_TUNE_VERSION > EARLIER
