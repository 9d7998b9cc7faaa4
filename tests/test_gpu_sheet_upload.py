"""Sheet uploads: the class map and representatives are checked and converted on the device; entries
out of range are refused as before, and the context stays usable."""
import numpy as np
import pytest

from pssfss_b200 import engine
from pssfss_b200.elements import rectstrip
from pssfss_b200.rwg import setup_rwg
from pssfss_b200.units import mm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field,index,value,message", [
    ("ufpm", 0, 0, "ufpm entry out of range"),
    ("ufpm", -1, 1 << 40, "ufpm entry out of range"),
    ("ufpm", 257, "nufp+1", "ufpm entry out of range"),
    ("ufp_rep", 0, 0, "ufp_rep out of range"),
    ("ufp_rep", -1, "pairs+1", "ufp_rep out of range"),
])
def test_out_of_range_classes_are_refused(field, index, value, message):
    sheet = rectstrip(Lx=4, Ly=4, Px=10, Py=10, Nx=3, Ny=5, units=mm)
    good, bad = setup_rwg(sheet), setup_rwg(sheet)
    arr = np.array(getattr(bad, field), np.int64, order="F")
    flat = arr.reshape(-1, order="A")
    flat[index] = {"nufp+1": bad.nufp + 1, "pairs+1": sheet.nface ** 2 + 1}.get(value, value)
    setattr(bad, field, flat.reshape(arr.shape, order="F"))
    with pytest.raises(RuntimeError, match=message):
        engine.face_integrals(sheet, bad, 1.0, 0.1, 0.2)
    assert np.isfinite(engine.face_integrals(sheet, good, 1.0, 0.1, 0.2)["J"]).all()
