"""The device scratch that the library reports for a call, and the serving
loop's estimate built on it (no device is needed)."""
from types import SimpleNamespace

import numpy as np

from xpsi_gb300 import batch as BT
from xpsi_gb300 import synthetic as SY
from xpsi_gb300._native import lib
from xpsi_gb300.serving import estimate_bytes

SMS = 152


def scratch(n=2, rows=200, cells=96, E=128, L=128, P=128, nmu=67, nE=166, mixed=0):
    return lib().xgpu_integrate_scratch_bytes(n, rows, cells, E, L, P, nmu, nE, mixed, 0, SMS)


def test_integrator_scratch_counts_every_part():
    # run records: 2 per SM of 36 bytes for each cell of a half and phase, twice
    runs = 2 * SMS * 2 * 48 * 128 * 36
    assert scratch() - scratch(mixed=1) == runs
    # none beyond 256 cells
    assert scratch(cells=257) == scratch(mixed=1)
    # one table slab per CTA
    assert scratch() - scratch(nmu=0, nE=0) == 2 * SMS * 67 * 166 * 8
    # a parallel more: its geometry records of two images, a chunk's partial
    more = scratch(rows=300) - scratch(rows=200)
    assert more >= 100 * (2 * 4 * 128 * 8 + 128 * 128 * 8)


def test_mesh_scratch_counts_every_part():
    n, S = 40, 96
    rows, cells = n * S, n * S * S
    b = lib().xgpu_mesh_scratch_bytes(n, rows, cells, S)
    table, edges, pieces = 8000, 5 * 8 * (S + 1), 4 * 128 * 8
    assert n * (table + edges + pieces) + rows * 10 * 8 + 8 * cells <= b
    # fewer than 5000 / 6 parallels queue no second list
    assert lib().xgpu_mesh_scratch_bytes(8, 8 * S, 8 * S * S, S) < b / 5 + 8 * 8 * S * S


def test_estimate_holds_the_scratch():
    m = SY.config2_model(K=20, q=16, num_energies=24, sqrt_num_cells=40, num_leaves=32,
                         num_rays=64, max_sqrt_num_cells=64, table_shape=(10, 8, 16, 60))
    rng = np.random.default_rng(1)
    P = BT.prepare(m, np.array([SY.prior_vector(rng) for _ in range(3)]), meshes="gpu")
    table = SimpleNamespace(nmu=16, nE=60)
    for precision, mixed in (("plain", 0), ("mixed", 1)):
        ev = SimpleNamespace(model=m, N_L=32, N_R=64, q=16, K=20, atmos=table, target_ctas=0,
                             sms=SMS, precision=precision)
        S_max = max(q.S1 for q in P.meshes)
        need = lib().xgpu_integrate_scratch_bytes(6, P.n_rows, S_max, 24, 32, 32, 16, 60, mixed, 0,
                                                  SMS)
        rays = 3 * P.n_rows * 64 * 8
        assert estimate_bytes(ev, P) > need + rays + P.n_cells * 36 + 6 * (24 + 16 + 20) * 32 * 8
