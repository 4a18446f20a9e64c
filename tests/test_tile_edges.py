"""The boundary kernels at sizes that leave remainders in every tile, against the FP64 oracle.

The free-surface kernel works in tiles of 16 columns x 4 planes, the fault band kernel in
tiles of 32 columns x 4 rows, the tiled volume kernels in tiles of 32 x 8 and 16 x 16 nodes,
the interior one with two neighbouring nodes per thread.  The grids below have 1, 13 and 15 columns left over
of 16, 1 to 3 planes of 4, fault rows that start and end inside a tile, and PML widths whose
edge falls inside a pair of nodes (in one of them the two y faces meet there); eight steps
run every operator direction of every stage.

Tolerances as in the parity tests of the same configurations (slip weakening in a layered
medium with PML and sponge 5e-4, rate and state on a rough fault 3e-3), relative to the
largest velocity and the largest stress.
"""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

GRIDS = [("sw", (45, 77, 47)), ("sw", (46, 81, 50)), ("sw", (51, 95, 53)), ("rs", (27, 79, 43))]


@pytest.mark.parametrize("law,size", GRIDS)
def test_remainders_match_oracle(oracle_lib, law, size):
    import dynfd3dcuda_b200 as dfd

    NX, NY, NZ = size
    if law == "sw":
        p, fx, st, layers, _, _ = cases.media_case(NX, NY, NZ, steps=8)
        tol, steps = 5e-4, 8
    else:
        p, fx, st, layers, _, _ = cases.rs_rough_case(NY, NX, NZ, seed=31, L=0.02, steps=16)
        p["smooth_load_T"] = 0.05
        tol, steps = 3e-3, 16
    sim = dfd.Simulation(p, fx, st, layers)
    o = oracle_lib.Oracle(p, fx, st, layers, double=True)
    sim.run(0, steps)
    for it in range(steps):
        o.step(it)
    sim.check_finite()
    W, Wo = sim.wave(), o.wave()
    for fields in (slice(0, 3), slice(3, 9)):
        scale = np.abs(Wo[fields]).max()
        assert scale > 0 and np.abs(W[fields] - Wo[fields]).max() < tol * scale, fields
    for names in (("slip",), ("Vs1", "Vs2"), ("Tn", "Ts1", "Ts2"), ("State",)):
        ref = [o.get(nm).reshape(NZ, NY) for nm in names]
        scale = max(np.abs(r).max() for r in ref)
        for nm, r in zip(names, ref):
            assert np.abs(sim.fault(nm) - r).max() <= tol * scale, nm


@pytest.mark.parametrize("size,pml", [((33, 47, 37), 11), ((41, 61, 34), 13), ((28, 22, 29), 11),
                                      ((36, 64, 40), 12)])
def test_pairs_across_face_edges(oracle_lib, size, pml):
    """Volume runs: odd and even y ends and PML widths, against the oracle (2e-5, as the
    volume parity cases)."""
    import dynfd3dcuda_b200 as dfd

    NX, NY, NZ = size
    p, fx, st, layers, _, _ = cases.get_case("vol_curved")
    p = dict(p, NX=NX, NY=NY, NZ=NZ, PML_N=pml)
    fx = cases.curved_geometry(NY, NZ, p["DH"], hill_amp=100.0, hill_width=600.0, seed=3)
    w0 = cases.smooth_wave(NX, NY, NZ, seed=4)
    sim = dfd.Simulation(dict(p, Rupture=0), fx, None, layers)
    sim.set_wave(w0.astype(np.float32))
    o = oracle_lib.Oracle(p, fx, st, layers, double=True)
    o.set("W", w0)
    sim.run(0, 8)
    for it in range(8):
        o.step_volume(it)
    W, Wo = sim.wave(), o.wave()
    for fields in (slice(0, 3), slice(3, 9)):
        scale = np.abs(Wo[fields]).max()
        assert scale > 0 and np.abs(W[fields] - Wo[fields]).max() < 2e-5 * scale, fields
