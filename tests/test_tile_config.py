"""The tile configuration can be saved and put back (host-side planning only)."""
import pytest

from nqpu_b200 import _lib, circuits
from nqpu_b200.state import Circuit

C128, C64 = 0, 1


def phase_estimation(n):
    return Circuit(n, [g for q in range(n) for g in (("h", (q,), ()), ("p", (q,), (0.1 * q + 0.2,)))] + circuits.qft(n))


@pytest.mark.parametrize("dtype,name", [(C64, "c64"), (C128, "c128")])
def test_save_set_restore(dtype, name):
    lib = _lib.load()
    # 27 qubits of phase estimation: the library takes complex64 tiles of 13 qubits
    # (7 passes), a setting of 4 would hold it to 12 (10 passes)
    c = phase_estimation(27)
    before = c.plan_stats(27, name, "tiled")
    saved = lib.nqpu_tile_config_get(dtype)
    for other in (1, 2, 4):
        assert lib.nqpu_tile_config_set(dtype, other) == 0
        assert lib.nqpu_tile_config_get(dtype) == other
        assert lib.nqpu_tile_config_set(dtype, saved) == 0
        assert lib.nqpu_tile_config_get(dtype) == saved
        assert c.plan_stats(27, name, "tiled") == before


@pytest.mark.parametrize("value", [3, 5, 8, 2**32 - 1])
def test_refused(value):
    lib = _lib.load()
    saved = lib.nqpu_tile_config_get(C64)
    assert lib.nqpu_tile_config_set(C64, value) == 2  # NQPU_INVALID_PARAMETER
    assert lib.nqpu_tile_config_get(C64) == saved


def test_default_is_the_library_choice():
    lib = _lib.load()
    assert lib.nqpu_tile_config_get(C64) == 0 and lib.nqpu_tile_config_get(C128) == 0
    c = phase_estimation(27)
    assert c.plan_stats(27, "c64", "tiled")["passes"] == 7
