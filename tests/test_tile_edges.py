"""The boundary kernels at sizes that leave remainders in every tile, against the FP64 oracle.

The free-surface kernel works in tiles of 16 columns x 4 planes, the fault band kernel in
tiles of 32 columns x 4 rows, the tiled volume kernels in tiles of 32 x 8 and 16 x 16 nodes,
the interior one with two neighbouring nodes per thread.  The grids below have 1, 13 and 15
columns left over of 16, 1 to 3 planes of 4, fault rows that start and end inside a tile and
odd and even PML widths (in one grid the two y faces meet, and no interior box is left); eight
steps run every operator direction of every stage.

A pair of the interior kernel with only one node to update has stores of its own.  With a PML
its box starts at a multiple of 16 in y and ends at a multiple of 4, so no pair hangs over its
end; two other edges split one:
  - the fault band, columns 30 .. NY - 32: with an even NY its last column is a pair's first
    node (NY = 94 and 78 below, where that column lies in the box);
  - the box's own end without a PML, where it holds every column and NY is odd.

Tolerances as in the parity tests of the same configurations (slip weakening in a layered
medium with PML and sponge 5e-4, rate and state on a rough fault 3e-3), relative to the
largest velocity and the largest stress.
"""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

GRIDS = [("sw", (45, 77, 47)), ("sw", (46, 81, 50)), ("sw", (51, 95, 53)), ("rs", (27, 79, 43)),
         ("sw", (51, 94, 53)), ("rs", (27, 78, 43))]


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


def check_volume(oracle_lib, size, over, rows=8):
    """Eight steps of a volume run against the oracle (2e-5, as the volume parity cases)."""
    import dynfd3dcuda_b200 as dfd

    NX, NY, NZ = size
    p, fx, st, layers, _, _ = cases.get_case("vol_curved")
    p = dict(p, NX=NX, NY=NY, NZ=NZ, **over)
    fx = cases.curved_geometry(NY, NZ, p["DH"], hill_amp=100.0, hill_width=600.0, seed=3)
    w0 = cases.smooth_wave(NX, NY, NZ, seed=4)
    sim = dfd.Simulation(dict(p, Rupture=0), fx, None, layers)
    sim.set_tile_rows(rows)
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


@pytest.mark.parametrize("size,pml", [((33, 47, 37), 11), ((41, 61, 34), 13), ((28, 22, 29), 11),
                                      ((36, 64, 40), 12)])
def test_remainders_around_faces(oracle_lib, size, pml):
    """Odd and even y ends and PML widths."""
    check_volume(oracle_lib, size, dict(PML_N=pml))


@pytest.mark.parametrize("rows", [8, 4])
@pytest.mark.parametrize("size,free", [((33, 47, 37), 1), ((28, 33, 29), 1), ((36, 65, 40), 0), ((24, 31, 27), 1)])
def test_half_pairs_at_the_box_end(oracle_lib, size, free, rows):
    """No PML and an odd NY: the last pair of every row holds one node (alone in its tile for
    33 and 65 columns), in both tile shapes of the interior kernel."""
    check_volume(oracle_lib, size, dict(usePML=0, FreeSurface=free), rows)
