"""``sweep_variant`` reads as a number that the library's entries take, also where
none was set, and reading it and putting it back changes nothing."""
import ctypes as C

import pytest


@pytest.fixture(params=["solver", "batch"])
def sim(pkg, monkeypatch, request):
    from starlab_physics_gb300 import solver

    monkeypatch.setattr(solver, "LBVH_CELL", lambda *a, **k: None)  # its constructor launches kernels
    x, f = pkg.grid_cloth(12)[:2]
    if request.param == "batch":
        inst = pkg.Instance(x, f, [], *pkg.box_mesh(0.5))
        return pkg.BatchedSolver([inst], 1.6e-5, 1e5, 1e8, (0, 0, -9.81), 1 / 60, device="cpu")
    return pkg.Solver(pkg.TriMesh(x, f, device="cpu"), None, 4e-6, 1e5, 1e8, (0, 0, -9.81), 1 / 60)


def test_reads_as_a_number(sim):
    from starlab_physics_gb300._lib import sx

    g, b = C.c_int(0), C.c_int(0)
    for sim.fast_math in (False, True):
        assert isinstance(sim.sweep_variant, int) and sim.sweep_variant == sim._default_variant[int(sim.fast_math)]
        sx.sx_jacobi_sweep_variant_info(sim.sweep_variant, C.addressof(g), C.addressof(b))
        assert g.value >= 1 and b.value >= 32


def test_put_back(sim):
    kept = sim.sweep_variant
    sim.sweep_variant = 5
    assert sim.sweep_variant == 5 and sim._sweep_variant == 5 and sim._packed_choice(1) == -1
    sim.sweep_variant = kept
    assert sim._sweep_variant is None
    sim.sweep_variant = int(kept)
    assert sim._sweep_variant == kept
    sim.sweep_variant = None
    assert sim._sweep_variant is None and sim.sweep_variant == kept
