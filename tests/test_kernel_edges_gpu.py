"""GPU kernels at the sizes where their splits, tiles and remainders change,
against the FP64 oracle or an explicit restatement in numpy."""
import numpy as np
import pytest

from apocharmm_b200 import api
from apocharmm_b200.systems import solvated_chain, water_box
from parity_util import oracle_for, rel_rms

pytestmark = pytest.mark.gpu

TIMFAC, KBOLTZ = 0.0488882129, 1.987191e-3
ATMOSP = 1.4584007e-05


# every radix (2 to 8) as first and as last stage, half spectra of odd and even
# length (nx / 2 + 1), one to several pencil slabs, planes of 256, 512 and 1,024
# threads; orders with and without the shared-memory patch
@pytest.mark.parametrize("nfft,order", [((16, 18, 20), 4), ((18, 16, 24), 6), ((20, 28, 30), 4),
                                        ((42, 40, 50), 6), ((50, 56, 36), 8), ((70, 40, 98), 4),
                                        ((64, 64, 64), 6), ((128, 100, 60), 4),
                                        ((90, 216, 32), 6), ((216, 180, 48), 4),
                                        # no room for the twiddles beside the plane
                                        ((256, 224, 16), 4), ((224, 252, 18), 6)])
def test_reciprocal_space_on_many_grids(tmp_path, nfft, order):
    s = water_box(300, 21.0, seed=9)
    st = dict(kappa=0.34, nfft=nfft, order=order, ctofnb=8.0, ctonnb=7.0, cutnb=9.0)
    psf, prm, fm, ctx = api.system_context(s, str(tmp_path), settings=st)
    fm.setComponentMask(4)
    ctx.calculateForces(False, True, False)
    E, G = oracle_for(s, st).evaluate(parts=("recip", "self"))
    # single-precision grids: 1e-6 of the gradient (5e-7 measured)
    assert rel_rms(ctx.getForces(), G) < 5e-6
    assert ctx.getPotentialEnergy() == pytest.approx(E["epot"], rel=1e-6)


@pytest.mark.parametrize("order", [4, 6, 8])
def test_reciprocal_space_of_atoms_far_apart(tmp_path, order):
    """Clusters whose grid points span more than the shared-memory patch take
    the points one by one: 20 waters (two clusters) in a 60 A box."""
    s = water_box(20, 60.0, seed=4, jitter=3.0)
    st = dict(kappa=0.34, nfft=(60, 64, 56), order=order, ctofnb=8.0, ctonnb=7.0, cutnb=9.0)
    psf, prm, fm, ctx = api.system_context(s, str(tmp_path), settings=st)
    fm.setComponentMask(4)
    ctx.calculateForces(False, True, False)
    E, G = oracle_for(s, st).evaluate(parts=("recip", "self"))
    assert rel_rms(ctx.getForces(), G) < 5e-6
    assert ctx.getPotentialEnergy() == pytest.approx(E["epot"], rel=1e-6)


# 1, 10, 11 and 21 waters fill one cluster or just leave it; 128 and 301 give
# work items whose last queue batch holds 1 to 32 atoms
@pytest.mark.parametrize("n", [1, 10, 11, 21, 128, 301])
@pytest.mark.parametrize("ron", [7.0, 8.0])
def test_direct_space_remainders(tmp_path, n, ron):
    L = max(18.5, (3 * n / 0.1003) ** (1.0 / 3.0))
    s = water_box(n, L, seed=n)
    st = dict(kappa=0.34, nfft=(20, 20, 20), order=4, ctofnb=8.0, ctonnb=ron, cutnb=9.0)
    psf, prm, fm, ctx = api.system_context(s, str(tmp_path), settings=st)
    fm.setComponentMask(2)
    E, G, W = oracle_for(s, st).evaluate(parts=("direct",), virial=True)
    # single-precision pairs: gradients to 1e-6 (2.3e-6 measured in these sparse
    # boxes); energies of up to about 20 kcal/mol a pair, each rounded at 6e-8,
    # cancel to tenths, so 1e-6 kcal/mol a pair; virial terms are some ten times
    # larger
    for energy, virial in ((False, False), (True, False), (True, True)):
        ctx.calculateForces(False, energy, virial)
        if n > 1:
            assert rel_rms(ctx.getForces(), G) < 5e-6
        if energy:
            assert ctx.getPotentialEnergy() == pytest.approx(E["epot"], rel=1e-6, abs=5e-6)
        if virial:
            assert np.abs(ctx.getVirial() - W).max() < 1e-6 * max(20.0, np.abs(W).max())


def test_default_work_items_of_a_large_box(tmp_path):
    """An i-atom's single-precision sum runs over a work item: its length does not
    grow with the system unless the caller asks for it."""
    n = 22000                                 # 66,000 atoms
    s = water_box(n, (3 * n / 0.1003) ** (1.0 / 3.0), seed=4)
    st = dict(kappa=0.34, nfft=(90, 90, 90), order=4, ctofnb=8.0, ctonnb=7.0, cutnb=9.0)
    g = {}
    for tiles in (None, 8, 16):
        keep = api.system_context(s, str(tmp_path / str(tiles)), settings=st, tiles_per_work=tiles)
        keep[2].setComponentMask(2)
        keep[3].calculateForces(False, False, False)
        g[tiles] = keep[3].getForces()
    assert np.array_equal(g[None], g[8])
    assert 0.0 < rel_rms(g[16], g[8]) < 1e-6


SMALL = 216     # waters: integrator kernels with four lanes a group
# more than 65,536 groups, of a water or of four free atoms: one lane a group,
# the direct-space grid that fills every SM
LARGE = 87500


def _water(n):
    """n waters and settings; thermostat and piston masses under which a step
    moves them alike at every n."""
    if n == SMALL:
        return (water_box(n, 19.0, seed=12),
                dict(kappa=0.34, nfft=(20, 20, 20), order=4, ctofnb=8.0, ctonnb=7.0, cutnb=9.0),
                2.0, 50.0)
    L = (3 * n / 0.1003) ** (1.0 / 3.0)
    return (water_box(n, L, seed=12),
            dict(kappa=0.34, nfft=(144, 144, 144), order=4, ctofnb=8.0, ctonnb=7.0, cutnb=9.0),
            2.0 * n / SMALL, 50.0 * (L / 19.0) ** 2)


def _flexible(tmp_path, dt, make, n=SMALL):
    s, st, nh_mass, _ = _water(n)
    keep = api.system_context(s, str(tmp_path), settings=st)
    fm, ctx = keep[2], keep[3]
    api.relax(ctx, None, iterations=60)
    ctx.useHolonomicConstraints(False)
    x = ctx.getCoordinates()
    v = np.random.default_rng(5).normal(size=x.shape) * np.sqrt(KBOLTZ * 500.0 / s.mass)[:, None]
    v -= (s.mass[:, None] * v).sum(0) / s.mass.sum()
    ctx.setVelocities(v)
    ctx.calculateForces(True, True, True)
    g, W = ctx.getForces(), ctx.getVirial()
    it = make(dt)
    it.setReferenceTemperature(300.0)
    it.setNoseHooverPistonMass(nh_mass)   # light: the passes differ by more than rounding
    it.setCharmmContext(ctx)
    it.propagate(1)
    return s, keep, it, x, v, g, W, dt / TIMFAC


@pytest.mark.parametrize("n", [SMALL, LARGE])
def test_nose_hoover_step_equals_explicit_passes(tmp_path, n):
    """One unconstrained step: the scalar predictor-corrector passes against
    three explicit passes over the atoms."""
    s, keep, it, x, v, g, W, h = _flexible(tmp_path, 0.001, api.CudaNoseHooverIntegrator, n)
    nh_mass = _water(n)[2]
    m = s.mass[:, None]
    p = h * v + 0.5 * h * h * g / m          # delta_prev from velocities and first forces,
    p -= (m * p).sum(0) / m.sum()            # without the drift, removed at step 0
    d = p - h * h * g / m
    ke_ref = 0.5 * keep[3].getDegreesOfFreedom() * KBOLTZ * 300.0

    def three(u):
        return ((0.5 * m * (p / h) ** 2).sum() + (0.5 * m * u ** 2).sum() + (0.5 * m * (d / h) ** 2).sum()) / 3.0

    ke, xi, pred = three(v), 0.0, d
    for k in range(3):
        f = 2.0 * h * (ke - ke_ref) / nh_mass
        xi = 0.0 + 0.5 * (f + (f if k == 0 else f0))
        f0 = f if k == 0 else f0             # the previous force starts as the first one
        u = (p + pred) / (2.0 * h)
        pred = d - h * h * xi * u
        ke = three(u)
    moved = np.abs(pred - d).max()
    assert moved > 1e-4                       # the thermostat matters in this step
    # forces evaluated twice differ by 1e-6 relative (list order): h^2 g / m of
    # a hydrogen at 1e2 kcal/mol/A is 4e-2 A, so 4e-8 A
    assert np.abs(keep[3].getCoordinates() - (x + pred)).max() < 2e-7
    assert np.abs(keep[3].getVelocities() - (pred + p) / (2.0 * h)).max() < 2e-7 / h


@pytest.mark.parametrize("passes,n", [(1, SMALL), (2, SMALL), (3, SMALL), (4, SMALL), (3, LARGE)])
def test_piston_step_equals_explicit_passes(tmp_path, passes, n):
    """One unconstrained cubic step without piston friction: box, coordinates
    and velocities against explicit passes over the atoms."""
    nh_mass, lp_mass = _water(n)[2:]

    def make(dt):
        it = api.CudaLangevinPistonIntegrator(dt)
        it.setCrystalType(it.CUBIC)
        it.setLangevinPistonMass([lp_mass])
        it.setMaxPredictorCorrectorIterations(passes)
        return it

    s, keep, it, x, v, g, W, h = _flexible(tmp_path, 0.001, make, n)
    fm, ctx = keep[2], keep[3]
    m = s.mass[:, None]
    p = h * v + 0.5 * h * h * g / m
    p -= (m * p).sum(0) / m.sum()   # the drift is removed at step 0
    d = p - h * h * g / m
    ke_ref = 0.5 * ctx.getDegreesOfFreedom() * KBOLTZ * 300.0
    L = s.box[0]
    V = L ** 3
    vfac = 1.0 / ATMOSP / V

    def kin(a):
        return np.einsum("ia,ib->ab", m * a, a) / (h * h)

    dp0 = vfac * (0.5 * (kin(d) + kin(p)) + W) - np.eye(3)
    static = dp0 - 0.25 * vfac * kin(d)
    dp = dp0
    ke = (0.5 * np.trace(kin(p)) + (0.5 * m * v ** 2).sum() + 0.5 * np.trace(kin(d))) / 3.0
    pred, r = d, x
    xx = r + d
    for k in range(passes):
        delta = (1.0 / lp_mass) * (np.trace(dp) / L) * V * h * h * ATMOSP
        onvel = 0.5 * delta / h
        pos = L + delta
        on, half = h * onvel / L, delta / (pos - 0.5 * delta)
        f = 2.0 * h * (ke - ke_ref) / nh_mass
        f0 = f if k == 0 else f0
        xi = 0.5 * (f + f0)
        u = (p + pred) / (2.0 * h)
        pred = d - (h * h * xi + h * on) * u
        xx = r + pred + half * 0.5 * (r + xx)
        dp = static + 0.25 * vfac * kin(pred)
        ke = (0.5 * np.trace(kin(p)) + (0.5 * m * u ** 2).sum() + 0.5 * np.trace(kin(pred))) / 3.0
    assert abs(delta) > 1e-5
    # the virial of the two evaluations differs by 1e-7 of its largest parts
    # (1e5 kcal/mol), 1e-2 kcal/mol: delta moves by h^2 / (50 L) of it, 5e-9 A
    assert fm.getBoxDimensions() == pytest.approx([pos] * 3, abs=2e-8)
    assert np.abs(ctx.getCoordinates() - xx).max() < 2e-7
    assert np.abs(ctx.getVelocities() - (pred + p) / (2.0 * h)).max() < 2e-7 / h


@pytest.mark.parametrize("kind", ["nose_hoover", "piston"])
def test_one_lane_a_group_holds_the_constraints(tmp_path, kind):
    s, st, _, _ = _water(LARGE)
    keep = api.system_context(s, str(tmp_path), settings=st)
    ctx = keep[3]
    w = api.water_indices(s)
    api.relax(ctx, w, iterations=60)
    ctx.assignVelocitiesAtTemperature(300.0)
    if kind == "piston":
        it = api.CudaLangevinPistonIntegrator(0.002)
        it.setCrystalType(it.CUBIC)
    else:
        it = api.CudaNoseHooverIntegrator(0.002)
    it.setReferenceTemperature(300.0)
    it.setCharmmContext(ctx)
    it.propagate(25)
    x, v = ctx.getCoordinates().reshape(-1, 3, 3), ctx.getVelocities()
    d = np.linalg.norm(x[:, [0, 0, 1]] - x[:, [1, 2, 2]], axis=2)
    # SETTLE works in FP64 on coordinates of up to 70 A: 1e-14 of them, squared
    # lengths of 1 A^2 to 1e-12
    assert np.abs(d - d[0]).max() < 1e-9
    drift = (s.mass[:, None] * v).sum(0) / np.abs(s.mass[:, None] * v).sum(0)
    # each force is rounded to 2^-40 kcal/mol/A, pairs are equal and opposite;
    # the reciprocal space leaves a net force of about 1e-5 of an atom's
    assert np.abs(drift).max() < 1e-4
    assert 200.0 < it.getInstantaneousTemperature() < 2000.0


def test_direct_space_of_a_large_box(tmp_path):
    """Work items of 8 and 16 tiles on a grid that fills every SM, against 64
    bits."""
    s, st, _, _ = _water(LARGE)
    for tiles in (8, 16):
        keep = api.system_context(s, str(tmp_path / str(tiles)), settings=st, tiles_per_work=tiles)
        fm, ctx = keep[2], keep[3]
        if tiles == 8:
            s.pos = api.relax(ctx, api.water_indices(s), iterations=40)
            E, G, W = oracle_for(s, st).evaluate(parts=("direct",), virial=True)
        fm.setComponentMask(2)
        for energy, virial in ((False, False), (True, True)):
            ctx.calculateForces(True, energy, virial)
            # 6.3e-7 to 7.7e-7 measured in larger and longer-ranged boxes
            assert rel_rms(ctx.getForces(), G) < 3e-6
        assert ctx.getPotentialEnergy() == pytest.approx(E["epot"], rel=1e-6)
        assert np.abs(ctx.getVirial() - W).max() < 1e-6 * np.abs(W).max()


def test_piston_virial_without_energies(tmp_path):
    """Within a segment the direct space leaves the energies out of the virial
    kernel; with one-step segments every step takes the kernel with both.  The
    lists differ (rebuilt every step or every 20), so single-precision sums
    differ by their rounding: 1e-7 of the virial, 1e-8 A of an edge in a step."""
    out = []
    for freq in (1, 20):
        s = water_box(600, 26.0, seed=8)
        st = dict(kappa=0.34, nfft=(28, 28, 28), order=4, ctofnb=9.0, ctonnb=8.0, cutnb=11.0)
        keep = api.system_context(s, str(tmp_path / f"f{freq}"), settings=st)
        fm, ctx = keep[2], keep[3]
        api.relax(ctx, api.water_indices(s), iterations=80)
        ctx.setRandomSeedForVelocities(3)
        ctx.assignVelocitiesAtTemperature(300.0)
        it = api.CudaLangevinPistonIntegrator(0.001)
        it.setCrystalType(it.CUBIC)
        it.setNonbondedListUpdateFrequency(freq)
        it.setCharmmContext(ctx)
        it.propagate(10)
        out.append((fm.getBoxDimensions(), ctx.getCoordinates(), ctx.getPotentialEnergy()))
    assert abs(out[0][0][0] - s.box[0]) > 1e-6
    assert out[0][0] == pytest.approx(out[1][0], abs=2e-7)
    assert np.abs(out[0][1] - out[1][1]).max() < 1e-5
    # the energies of the last step are there either way
    assert out[0][2] == pytest.approx(out[1][2], rel=1e-5)
    assert abs(out[1][2]) > 100.0


@pytest.mark.parametrize("steps", [1, 25])
def test_piston_leaves_the_last_forces(tmp_path, steps):
    """After a piston run the context holds the gradient of its last
    evaluation, as it holds that evaluation's energies and virial."""
    s = water_box(216, 19.0, seed=12)
    st = dict(kappa=0.34, nfft=(20, 20, 20), order=4, ctofnb=8.0, ctonnb=7.0, cutnb=9.0)
    keep = api.system_context(s, str(tmp_path), settings=st)
    ctx = keep[3]
    api.relax(ctx, api.water_indices(s), iterations=60)
    ctx.assignVelocitiesAtTemperature(300.0)
    it = api.CudaLangevinPistonIntegrator(0.001)
    it.setCrystalType(it.CUBIC)
    it.setCharmmContext(ctx)
    if steps > 1:
        it.propagate(steps - 1)
    ctx.calculateForces(True, True, True)
    g, e, w = ctx.getForces(), ctx.getEnergyComponents(), ctx.getVirial()
    it.propagate(1)
    # the same coordinates and box, a list built again: sums in another order
    assert rel_rms(ctx.getForces(), g) < 1e-5
    assert ctx.getEnergyComponents() == pytest.approx(e, rel=1e-5, abs=1e-3)
    assert np.abs(ctx.getVirial() - w).max() < 1e-5 * np.abs(w).max()
    # and within a longer segment: the last step's, not an earlier one's or none
    it.propagate(3)
    last = ctx.getForces()
    assert np.abs(last).max() > 1.0 and rel_rms(last, g) > 1e-5


@pytest.mark.parametrize("restraint", [False, True])
def test_steps_of_forces_alone_leave_the_energy_slots_clear(tmp_path, restraint):
    """Only the first step of a segment clears the energy slots, plug-in forces or
    not; with one-step segments every step does."""
    out = []
    for freq in (1, 20):
        s = water_box(600, 26.0, seed=8)
        st = dict(kappa=0.34, nfft=(28, 28, 28), order=4, ctofnb=9.0, ctonnb=8.0, cutnb=11.0)
        keep = api.system_context(s, str(tmp_path / f"f{freq}"), settings=st)
        ctx = keep[3]
        api.relax(ctx, api.water_indices(s), iterations=20)
        ctx.assignVelocitiesAtTemperature(300.0)
        if restraint:
            hold = api.HarmonicRestraintForce(s.n_atoms)
            hold.setReferenceCoordinates(ctx.getCoordinates() + 0.1)
            hold.setSelection(np.arange(3))
            hold.setForceConstant(1.0)
            keep[2].subscribe(hold, "hold")
        it = api.CudaLangevinThermostatIntegrator(0.001)
        it.setNonbondedListUpdateFrequency(freq)
        it.setCharmmContext(ctx)
        assert abs(ctx.calculatePotentialEnergy(True)) > 100.0
        held = ctx.getEnergyComponent("hold") if restraint else 0.0
        it.propagate(6)
        out.append(ctx.getEnergyComponents())
        # all but the self energy, which is no slot; the plug-in's own slot keeps
        # its last evaluated energy
        assert all(v == 0.0 for k, v in out[-1].items() if k != "ewse")
        if restraint:
            assert ctx.getEnergyComponent("hold") == held > 0.0
    assert out[0] == out[1]
