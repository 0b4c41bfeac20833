"""The dense Davidson near convergence: sweep energies stay variational.

Transverse-field Ising on the 6 x 12 cylinder (dense path, no quantum numbers), a
seeded random product start, six sweeps.  From the third sweep on every energy is
within 1e-4 of the ground state's and the state changes little, so no sweep may come
out above the one before it by more than its own accuracy (1e-8 per site): a new
direction that is nearly parallel to the earlier ones used to enter the projected
matrix without being orthogonal to them (linalg/tensor_davidson.cpp:74-184 projects
once), and a converged sweep then reported up to 5e-3 too much.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [12, 13])
def test_sweep_energies_do_not_rise(seed):
    import tt_b200
    from oracle import autompo as am
    Nx, Ny, g = 12, 6, 3.0
    N = Nx * Ny
    a = tt_b200.AutoMPO()
    for s1, s2, *_ in am.snake_relabel(am.square_lattice(Nx, Ny, True), Nx, Ny):
        a.add(-4.0, "Sz", s1 - 1, "Sz", s2 - 1)
    for i in range(N):
        a.add(-2.0 * g, "Sx", i)
    ctx = tt_b200.Context(0)
    try:
        psi = tt_b200.DMPS(N, list(np.random.default_rng(seed).integers(0, 2, N)))
        H = tt_b200.DMPO.from_autompo(a, N)
        _, sweeps, _ = tt_b200.ddmrg_run(psi, H, 6, [16, 32, 64, 128, 128, 128], [1e-10], [4])
        del psi, H
    finally:
        ctx.close()
    assert np.all(np.diff(sweeps) <= 1e-8 * N), sweeps
