"""The staging of the a-trous passes can be set to every mode and back to the default one, and to no other."""
import pytest

from photon_b200 import abi, native

pytestmark = pytest.mark.gpu


def test_a_session_returns_to_the_default_staging():
    s = native.Svgf(64, 48)
    for mode in (0, 1, 2, 3, 4):
        s.set_tma(mode)
    for mode in (-1, 5):
        with pytest.raises(native.PhotonError) as e:
            s.set_tma(mode)
        assert e.value.code == abi.PT_ERR_INVALID
    s.close()
