"""A workspace size may be asked for no rows; the gradient itself refuses them."""
import ctypes

import pytest

from flowmc_gb300 import _lib
from test_train_workspace import SHAPES, _flow, _size

pytestmark = pytest.mark.skipif(not _lib.LIB_PATH.exists(), reason="libflowmc.so not built")


@pytest.mark.parametrize("d,L,hidden,nb,prec", SHAPES)
def test_no_rows(d, L, hidden, nb, prec):
    s = _flow(d, L, hidden, nb, getattr(_lib, f"PREC_{prec}"))
    assert _size(s, 0) >= 0   # an answer, not a division by zero
    assert _lib.lib().fmc_flow_loss_grad(ctypes.byref(s), 256, 0, 256, 256, 256, 1 << 30, None) != 0
    assert "n=0 < 1" in _lib.lib().fmc_last_error().decode()
