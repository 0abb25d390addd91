"""The Schwarz factors of a geometry, bit for bit, whatever the handle did before: on a new handle, when the
same geometry is set again, after a different one, and under another schedule.  Each factor is the
largest of a quartet's own integrals, computed by one thread or one warp in a fixed order.
"""
import numpy as np
import pytest

from hfscf_b200 import basis as B
from hfscf_b200 import engine as E
from hfscf_b200 import molecules as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["6-31g**", "cc-pvdz"])
def test_schwarz_factors_do_not_depend_on_the_handles_history(name):
    # long contractions and many pairs: the (dp|dp) class of its lists is above the limit of the small builds
    Z, x = M.n_alkane(7)
    x = np.asarray(x) * B.ANGSTROM_TO_BOHR
    bs = B.build_basis(name, Z, x, pure=name == "cc-pvdz")
    with E.Engine(bs) as eng:
        first = eng.schwarz()
        eng.set_geometry(x)
        again = eng.schwarz()
        eng.set_geometry(30.0 * x)  # next to no quartets
        eng.set_geometry(x)
        after = eng.schwarz()
        eng.set_schedule(np.tile(np.array((32, 0, 0, 1), dtype=np.int32), (E.NUM_CLASSES, 1)))
        eng.set_geometry(x)
        scheduled = eng.schwarz()
    assert np.array_equal(first, again)
    assert np.array_equal(first, after)
    assert np.array_equal(first, scheduled)
