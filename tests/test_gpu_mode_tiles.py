"""Elements without 3-D properties run in tiles of modes (solid1d_kernel.cuh): parity with the FP64
oracle at the edges of the tiles -- one mode, a full tile, one mode more, several uneven tiles --
for the block sizes that axg_set_team_size allows, on the axis and off it, and with batched
wavefields split over blocks.

Tolerances: a force is a sum of about 1e2 products, each operand rounded once, so its relative
2-norm error is a few units of the working precision: 2e-6 in float, 1e-13 in double.
"""
import numpy as np
import pytest

from axisem3d_b200 import meshgen
from axisem3d_b200.solver import Solver

pytestmark = pytest.mark.gpu

TOL = {"fp32": 2e-6, "mixed": 2e-6, "fp64": 1e-13}


def _oracle_steps(m, u, n):
    import oracle as O
    o = O.Oracle(m, "fp64", threads=4)
    o.set_field(u, "displ")
    o.compute_stiffness()
    f = o.get_field("stiff")
    o2 = O.Oracle(m, "fp64", threads=4)
    o2.set_field(u, "displ")
    o2.run(n)
    return f, o2.get_field("displ")


@pytest.mark.parametrize("precision", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("nrs", [[1], [1, 2, 3], [8, 9], [9, 10, 11], [20, 21], [63, 64]])
@pytest.mark.parametrize("team", [0, 32, 256])
def test_tiles_match_oracle(built, precision, nrs, team):
    m = meshgen.microbench_model(n_elem=12, nr_choices=nrs, is3d=False, axial_column=True, seed=3)
    u = meshgen.random_displacement(m, seed=4)
    f, d = _oracle_steps(m, u, 4)
    teams = {c: team for c in range(5)} if team else None
    with Solver(m, precision, team_sizes=teams) as s:
        s.set_field(u, "displ")
        s.compute_stiffness()
        g = s.get_field("stiff")
        assert np.linalg.norm(g - f) <= TOL[precision] * np.linalg.norm(f)
    with Solver(m, precision, team_sizes=teams) as s:
        s.set_field(u, "displ")
        s.run(4)
        assert np.linalg.norm(s.get_field("displ") - d) <= TOL[precision] * np.linalg.norm(d)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("nr", [1, 2, 9, 11, 12, 40])
def test_cg4_tiles_match_oracle(built, precision, nr):
    """CG4: the recursion runs on threads of its own, one per (component, attenuating slot)."""
    m = meshgen.microbench_model(n_elem=9, nr_choices=[nr], is3d=False, rheology="iso", attenuation="cg4", seed=5)
    u = meshgen.random_displacement(m, seed=6)
    f, d = _oracle_steps(m, u, 5)
    with Solver(m, precision) as s:
        s.set_field(u, "displ")
        s.compute_stiffness()
        assert np.linalg.norm(s.get_field("stiff") - f) <= TOL[precision] * np.linalg.norm(f)
    with Solver(m, precision) as s:
        s.set_field(u, "displ")
        s.run(5)
        assert np.linalg.norm(s.get_field("displ") - d) <= TOL[precision] * np.linalg.norm(d)


@pytest.mark.parametrize("nwave", [2, 7])
def test_waves_split_over_blocks(built, nwave):
    """Few elements and several wavefields: each wavefield equals its own run."""
    m = meshgen.microbench_model(n_elem=4, nr_choices=[9, 11], is3d=False, seed=7)
    us = [meshgen.random_displacement(m, seed=10 + w) for w in range(nwave)]
    one = []
    for u in us:
        with Solver(m, "fp64") as s:
            s.set_field(u, "displ")
            s.run(5)
            one.append(s.get_field("displ"))
    m.nwave = nwave
    with Solver(m, "fp64") as s:
        s.set_field(np.concatenate(us), "displ")
        s.run(5)
        got = s.get_field("displ").reshape(nwave, -1)
    for w in range(nwave):
        assert np.linalg.norm(got[w] - one[w]) <= 1e-13 * np.linalg.norm(one[w])


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("attenuation, nrs", [("full", [9, 17, 30, 34]), ("full", [70, 96]), ("cg4", [64])])
def test_attenuating_slices_split_over_blocks(built, attenuation, nrs, precision):
    """The same for 3-D elements with attenuation: every wavefield of a batch has its own memory
    variables."""
    nwave = 5
    m = meshgen.microbench_model(n_elem=6, nr_choices=nrs, attenuation=attenuation, seed=7)
    us = [meshgen.random_displacement(m, seed=10 + w) for w in range(nwave)]
    one = []
    for u in us:
        with Solver(m, precision) as s:
            s.set_field(u, "displ")
            s.run(4)
            s.compute_stiffness()
            one.append((s.get_field("displ"), s.get_field("stiff")))
    m.nwave = nwave
    with Solver(m, precision) as s:
        s.set_field(np.concatenate(us), "displ")
        s.run(4)
        s.compute_stiffness()
        got = [s.get_field(k).reshape(nwave, -1) for k in ("displ", "stiff")]
    for w in range(nwave):
        for g, ref in zip(got, one[w]):
            assert np.linalg.norm(g[w] - ref) <= TOL[precision] * np.linalg.norm(ref)


def test_handles_of_two_precisions_share_kernels(built):
    """FP32 and mixed handles launch the same fluid kernels: a small handle of one precision must
    not lower the shared-memory limit that a large one of the other has raised."""
    large = meshgen.spherical_model(n_theta=24, n_solid_layers=3, n_fluid_layers=1, nr_min=125, nr_max=125)
    small = meshgen.spherical_model(n_theta=8, n_solid_layers=2, n_fluid_layers=1, nr_min=81, nr_max=81)
    for precision, other in (("mixed", "fp32"), ("fp32", "mixed")):
        with Solver(large, precision) as s:
            s.run(2)
        with Solver(small, other) as s:
            s.run(2)
        with Solver(large, precision) as s:
            s.run(2)
            assert np.all(np.isfinite(s.get_field("displ")))


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("nrs", [
    [26, 27], [28, 30, 32], [33, 35, 36], [39, 40, 42, 44], [45, 48, 49, 50], [52, 54, 55, 56], [60, 63, 64, 65],
    [66, 70, 72, 75, 77], [78, 80, 81, 84, 88], [90, 91, 96, 98, 99], [100, 104, 105, 108, 110],
    [112, 117, 120, 121], [125, 126, 128], [29, 31, 34, 37, 58, 61]])
@pytest.mark.parametrize("attenuation", [None, "full"])
def test_slice_transforms_match_oracle(built, precision, nrs, attenuation):
    """3-D elements of every nr from 26 on: FFTs where nr has no prime factor above 13 (every radix
    and every pair of radices of two-pass transforms, three passes), direct sums for the others."""
    m = meshgen.microbench_model(n_elem=9, nr_choices=nrs, rheology="iso", attenuation=attenuation, seed=nrs[0])
    u = meshgen.random_displacement(m, seed=8)
    f, d = _oracle_steps(m, u, 3)
    with Solver(m, precision) as s:
        s.set_field(u, "displ")
        s.compute_stiffness()
        g = s.get_field("stiff")
        assert np.linalg.norm(g - f) <= TOL[precision] * np.linalg.norm(f)
    with Solver(m, precision) as s:
        s.set_field(u, "displ")
        s.run(3)
        assert np.linalg.norm(s.get_field("displ") - d) <= TOL[precision] * np.linalg.norm(d)


@pytest.mark.parametrize("nr", [26, 100])
def test_cg4_slices_match_oracle(built, nr):
    """CG4 on slices: the attenuating points run apart from the elastic ones, also where a chunk of
    the slice phase holds only some of them."""
    m = meshgen.microbench_model(n_elem=6, nr_choices=[nr], attenuation="cg4", seed=9)
    u = meshgen.random_displacement(m, seed=8)
    f, d = _oracle_steps(m, u, 4)
    for teams in (None, {3: 128, 4: 128}):
        with Solver(m, "mixed", team_sizes=teams) as s:
            s.set_field(u, "displ")
            s.compute_stiffness()
            assert np.linalg.norm(s.get_field("stiff") - f) <= TOL["mixed"] * np.linalg.norm(f)
        with Solver(m, "mixed", team_sizes=teams) as s:
            s.set_field(u, "displ")
            s.run(4)
            assert np.linalg.norm(s.get_field("displ") - d) <= TOL["mixed"] * np.linalg.norm(d)


@pytest.mark.parametrize("pieces", [[64], [1, 7, 8, 48], [15, 16, 17, 16], [33, 31]])
def test_step_graphs_of_one_and_several_steps(built, pieces):
    """Runs of any length replay captured steps: the same steps, records and source times as launch by
    launch."""
    m = meshgen.cartesian_model(nx=7, nz=5, nr=5, nstations=4, record_interval=3)
    with Solver(m, "fp64") as s:
        s.run(64, graph=False)
        ref, seis = s.get_field("displ"), s.seismograms()
    with Solver(m, "fp64") as s:
        for n in pieces:
            s.run(n)
        assert s.step == 64
        d, g = s.get_field("displ"), s.seismograms()
    assert np.linalg.norm(d - ref) <= 1e-12 * np.linalg.norm(ref)
    assert g.shape == seis.shape and np.linalg.norm(g - seis) <= 1e-12 * np.linalg.norm(seis)


def test_more_wavefields_than_one_grid_axis(built):
    """A wavefield beyond the 32768 rows of the point update's second grid axis is updated too."""
    m = meshgen.microbench_model(n_elem=1, nr_choices=[1], is3d=False, rheology="iso", attenuation=None, seed=3)
    u = meshgen.random_displacement(m, seed=4)
    with Solver(m, "fp32") as s:
        s.set_field(u, "displ")
        s.run(3)
        one = s.get_field("displ")
    m.nwave = 32770
    full = np.zeros((m.nwave, u.size), np.complex128)
    full[0] = full[-1] = u
    with Solver(m, "fp32") as s:
        s.set_field(full.ravel(), "displ")
        s.run(3)
        got = s.get_field("displ").reshape(m.nwave, -1)
    assert not np.any(got[1:-1])
    for w in (0, -1):
        assert np.linalg.norm(got[w] - one) <= 1e-6 * np.linalg.norm(one)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_small_buckets_largest_elements_first(built, precision):
    """A bucket of about one wave of blocks runs in the order of falling nr: state, moduli and
    offsets follow their elements, step after step."""
    m = meshgen.microbench_model(n_elem=40, nr_min=26, nr_max=64, seed=17)
    u = meshgen.random_displacement(m, seed=8)
    f, d = _oracle_steps(m, u, 4)
    with Solver(m, precision) as s:
        s.set_field(u, "displ")
        s.compute_stiffness()
        assert np.linalg.norm(s.get_field("stiff") - f) <= TOL[precision] * np.linalg.norm(f)
    with Solver(m, precision) as s:
        s.set_field(u, "displ")
        s.run(4)
        assert np.linalg.norm(s.get_field("displ") - d) <= TOL[precision] * np.linalg.norm(d)
