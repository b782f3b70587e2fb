"""The adjoint kernel's two forms (the one for short chunks skips what the
pipeline fill's planes compute for nobody) and the imaging kernel, which
always skips it, give the same images whatever the chunk: chunks of one and
two planes, at the limit between the forms, of a whole column, and a
top/bottom split of each form; with every precision of the stored snapshots,
whose planes above the free surface imaging mirrors itself."""
import numpy as np
import pytest

import miniappsforhpe_b200 as P
from miniappsforhpe_b200 import earth_models as EM

NX, NY, NZ, NT = 40, 19, 80, 24
SPLITS = ((80, 0), (64, 0), (65, 0), (1, 0), (2, 0), (5, 70), (9, 12))


@pytest.mark.gpu
@pytest.mark.parametrize("snap", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("fs", [True, False], ids=["fs", "nofs"])
@pytest.mark.parametrize("tti", [True, False], ids=["tti", "vti"])
def test_chunk_length_does_not_change_images(tti, fs, snap):
    model = (EM.smooth_tti(NX, NY, NZ, corr_m=60.0, seed=3) if tti else EM.layered_vti(NX, NY, NZ, seed=3))
    dt = EM.cfl_dt(model, 10.0)
    first = None
    try:
        for bz, zt in SPLITS:
            for k in ("adjoint", "imaging"):
                P.tune_set(NX, NY, NZ, k, bz, zt)
            with P.Simulator(P.Config(nx=NX, ny=NY, nz=NZ, dt=dt, nt=NT, sponge_width=6, free_surface=fs,
                                      snap_precision=snap)) as sim:
                sim.set_model(**model)
                sim.set_source(NX // 2, NY // 2, 5, EM.ricker(NT, dt, 40.0) * 1e3)
                sim.set_receivers(EM.receiver_plane(NX, NY, 3))
                sim.adjoint(sim.forward())
                out = sim.image()
            first = first or out
            for a, b in zip(out, first):
                assert np.abs(b).max() > 0
                np.testing.assert_array_equal(a, b)
    finally:
        for k in P.TUNE_KINDS:
            P.tune_set(NX, NY, NZ, k, 0)
