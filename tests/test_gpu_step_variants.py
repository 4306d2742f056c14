"""The step kernel over its variants: 8, 16 and 32 lanes per particle, with and
without energies, switched and plain cutoff, both precisions, and the walks by
the axes that take the minimum image.  Forces against the FP64 oracle over the
particles near each combination of faces (the walk of x and y alone among them),
within the 5e-5 relative RMS stated for FP32 boxes."""
import numpy as np
import pytest

from conftest import relrms
from oracle import pyoracle as po
from quantom_b200 import engine as E
from quantom_b200 import systems as S

pytestmark = pytest.mark.gpu


# 32 lanes (with energies too), 16 and 8
@pytest.mark.parametrize("box,waters", [(3.0, 881), (4.6, 3201), (6.0, 7103)])
@pytest.mark.parametrize("switch_on", [0.8, 1.0])   # the cutoff is 1.0
@pytest.mark.parametrize("precision", [0, 1])
def test_forces_by_faces(box, waters, switch_on, precision):
    spec = S.SystemSpec("box", box, waters, cutoff=1.0, mc_sweeps=10)
    s = S.make_system(spec, seed=31)
    x = np.mod(s.solvents["pos"].astype(np.float64), box).astype(np.float32)
    s.solvents["pos"] = x
    s.solvents["pos_tsub1"] = x
    F64, _ = po.PhysSystem(s, rc=1.0, r_on=switch_on).forces(x.astype(np.float64))
    p = E.default_params(box_len=box, cutoff=1.0, dt=spec.dt, semantics=E.SEMANTICS_PHYSICS, skin=0.1,
                         switch_on=switch_on, nlist_period=10, precision=precision)
    near = ((x < 1.0) | (x > box - 1.0)) @ np.array([1, 2, 4])
    with E.Engine(s, p) as eng:
        eng.compute_energies()
        _, with_energies = eng.forces()
        eng.step(1)                       # the same positions, without energies
        _, plain = eng.forces()
    for mask in range(8):
        m = near == mask
        assert m.sum() > 3, mask
        assert relrms(with_energies[m], F64[m]) < 5e-5, mask
        assert relrms(plain[m], F64[m]) < 5e-5, mask
