"""The loss and adjoint pair kernels over their variants: 8 and 16 lanes per
particle, 16- and 32-bit list ids, one and several types, one to the most bins.
Occupancies within 1e-5 of the FP64 oracle's (as tests/test_gpu_grad.py) and
gradients within 1e-3 relative of central differences of its loss."""
import numpy as np
import pytest

from quantom_b200 import engine as E
from quantom_b200 import systems as S

pytestmark = pytest.mark.gpu


def _box(box, waters, chains=0, length=0):
    spec = S.SystemSpec("box", box, waters, chains=S.ChainSpec(chains, length) if chains else None, mc_sweeps=4)
    s = S.make_system(spec, seed=21)
    p = dict(box_len=box, cutoff=1.2, dt=spec.dt, semantics=E.SEMANTICS_PHYSICS, skin=0.2, switch_on=1.0,
             nlist_period=0)
    with E.Engine(s, E.default_params(thermostat=E.THERMOSTAT_BERENDSEN, t_target=300.0, **p)) as eng:
        eng.step(200)   # off the packing's contacts
        s = s.with_state(*eng.compound_states(), eng.solvents())
    return s, E.default_params(**p)


@pytest.mark.parametrize("bins", [1, 7, 50, 128])
@pytest.mark.parametrize("box,waters,chains", [(3.1, 901, 0), (6.0, 6200, 2)])
def test_occupancies_match_fp64(bins, box, waters, chains):
    from oracle import pyoracle as po
    s, p = _box(box, waters, chains, 24)
    r_max = 1.2 * bins / (bins + 1) * 0.999
    with E.Engine(s, p) as eng:
        h = eng.rdf(bins, r_max)
    want = po.PhysSystem(s, rc=1.2, r_on=1.0).rdf(bins, r_max)
    assert np.abs(h - want).max() < 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("box,waters,chains", [(4.0, 1901, 2),      # 16 lanes, five types
                                               (6.0, 6143, 0),      # 16 lanes, one type
                                               (6.0, 6200, 0),      # 8 lanes
                                               (6.0, 6150, 2),      # 8 lanes, five types
                                               (13.0, 66003, 0)])   # 32-bit ids
def test_gradient_matches_fp64_differences(box, waters, chains):
    from oracle import pyoracle as po
    s, p = _box(box, waters, chains, 24)
    bins, steps = 20, 3
    r_max = 1.2 * bins / (bins + 1) * 0.999
    ps = po.PhysSystem(s, rc=1.2, r_on=1.0)
    target = 0.97 * ps.rdf(bins, r_max)
    with E.Engine(s, p) as eng:
        loss, g = eng.grad(steps, 2, bins, r_max, 1.0, 100.0, target)
    th = ps.params()
    value = lambda t: ps.with_params(t).loss(s.spec.dt, steps, bins, r_max, 1.0, 100.0, target)[0]  # noqa: E731
    assert abs(loss - value(th)) < 1e-5 * abs(loss)
    n_types = len(np.unique(np.concatenate([[0], s.compounds["atom_types"].ravel()]))) if chains else 1
    for k in (0, n_types):   # sigma and epsilon of the waters
        e = np.zeros(len(th))
        e[k] = 1e-4 * abs(th[k])
        fd = (value(th + e) - value(th - e)) / (2 * e[k])
        assert abs(g[k] - fd) < 1e-3 * abs(fd), (k, g[k], fd)


@pytest.mark.parametrize("bins", [75, 76, 77])
def test_bins_around_the_plain_shared_memory_limit(bins, tmp_path):
    """The loss kernel's columns of 76 bins and its static arrays together pass
    the 48 KB a launch gets unasked.  Each count in a process of its own: a
    larger count would raise the kernel's limit for those after it."""
    import subprocess
    import sys
    from conftest import ROOT
    code = ("from quantom_b200 import engine as E, systems as S\n"
            "s = S.make_system('tiny_solvent', seed=3)\n"
            "p = E.default_params(box_len=s.spec.box_len, cutoff=s.spec.cutoff, dt=s.spec.dt, "
            "semantics=E.SEMANTICS_PHYSICS, skin=0.1, switch_on=1.0, nlist_period=0)\n"
            f"h = E.Engine(s, p).rdf({bins}, 1.0)\n"
            "assert h.sum() > 0\n")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_threads_with_different_bins():
    """Engines on eight host threads whose loss kernels need two different amounts
    of shared memory beyond the plain limit: no launch is refused."""
    import threading
    s = S.make_system("tiny_solvent", seed=3)
    p = E.default_params(box_len=s.spec.box_len, cutoff=s.spec.cutoff, dt=s.spec.dt, semantics=E.SEMANTICS_PHYSICS,
                         skin=0.1, switch_on=1.0, nlist_period=0)
    failed = []

    def run(bins):
        with E.Engine(s, p) as eng:
            for _ in range(3000):
                try:
                    eng.rdf(bins, 1.0)
                except E.LimaError as e:
                    failed.append((bins, str(e)))
                    return

    threads = [threading.Thread(target=run, args=(b,)) for b in (128, 77) * 4]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


@pytest.mark.parametrize("bins", [1, 50])
def test_occupancies_do_not_depend_on_the_particle_order(bins):
    """Occupancies are exact sums of the pairs' weights (integers in units of
    2^-32; with 4,096 particles every partial sum is exact in FP64 too): the same
    box with its waters in another order gives the same bits.  One bin takes the
    32-bit columns past 2^32 many times."""
    from dataclasses import replace
    s = S.make_system("lj_solvent_4096", seed=3)
    p = E.default_params(box_len=s.spec.box_len, cutoff=s.spec.cutoff, dt=s.spec.dt, semantics=E.SEMANTICS_PHYSICS,
                         skin=0.1, switch_on=1.0, nlist_period=0)
    order = np.random.default_rng(8).permutation(s.n_solvents)
    h = []
    for t in (s, replace(s, solvents=s.solvents[order].copy())):
        with E.Engine(t, p) as eng:
            h.append(eng.rdf(bins, 1.2 * bins / (bins + 1) * 0.999))
    assert np.array_equal(h[0], h[1])


@pytest.mark.parametrize("box,waters,entries", [(4.0, 1901, 2),      # 16 lanes
                                                (6.0, 6150, 2),      # 8 lanes
                                                (13.0, 66003, 1)])   # 32-bit ids
def test_gradient_of_a_chain_type(box, waters, entries):
    """The derivatives that land on another type than the waters' (in the lane's
    own columns): sigma and epsilon of the last chain type."""
    from oracle import pyoracle as po
    s, p = _box(box, waters, 2, 24)
    bins, steps = 20, 2
    r_max = 1.2 * bins / (bins + 1) * 0.999
    ps = po.PhysSystem(s, rc=1.2, r_on=1.0)
    target = 0.97 * ps.rdf(bins, r_max)
    with E.Engine(s, p) as eng:
        _, g = eng.grad(steps, 2, bins, r_max, 1.0, 100.0, target)
        n_types = eng.param_layout()["n_types"]
    th = ps.params()
    value = lambda t: ps.with_params(t).loss(s.spec.dt, steps, bins, r_max, 1.0, 100.0, target)[0]  # noqa: E731
    kind = int(s.compounds[0]["atom_types"][: s.compounds[0]["n_particles"]].max())
    assert kind > 0
    for k in (kind, n_types + kind)[:entries]:
        e = np.zeros(len(th))
        e[k] = 1e-4 * abs(th[k])
        fd = (value(th + e) - value(th - e)) / (2 * e[k])
        assert abs(g[k] - fd) < 1e-3 * abs(fd), (k, g[k], fd)
