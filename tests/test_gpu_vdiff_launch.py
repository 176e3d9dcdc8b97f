"""The implicit vertical diffusion of the FP32 step as the update's epilogue or as its own launch, which the
depth of the mesh decides until it is set: the same bits whichever runs, on either side of the line."""
import numpy as np
import pytest

from fesom2_gb300 import gpu as G
from fesom2_gb300 import mesh as M
from oracle import oracle as O

pytestmark = pytest.mark.gpu


# own launch from 65 layers with groups of 2 slots, from 56 with groups of 4
@pytest.mark.parametrize("layers,width,own", [(64, 2, False), (65, 2, True), (128, 2, True), (55, 4, False),
                                              (56, 4, True), (128, 4, True)])
def test_either_launch_gives_the_same_bits(layers, width, own):
    ntr = 3
    mesh = M.channel_mesh(20, 23, 5000.0, M.stretched_zbar(layers, 10.0, 100.0))
    f = O.ensure_f64(M.make_forcing(mesh, "channel", seed=3, dt=600.0))
    val = [np.ascontiguousarray(t, dtype=np.float64) for t in M.make_tracers(mesh, "channel", ntr=ntr, seed=4)]
    got, launches = [], []
    for variant in (None, 0, 2):
        ctx = G.Context(mesh, G.PREC_FP32, max_tracers=ntr)
        ctx.set_tracer_width(width)
        if variant is not None:
            ctx.set_stage_variant(3, variant)
        ctx.state_setup([G.tra_cfg(id=k + 1) for k in range(ntr)])
        ctx.forcing_upload(f)
        for k in range(ntr):
            ctx.tracer_upload(k, val[k], 0.999 * val[k])
        ctx.run_steps(f.dt, 2)
        got.append([ctx.tracer_download(k) for k in range(ntr)])
        launches.append(ctx.launches_per_step())
        ctx.close()
    assert launches[2] == launches[1] + 1
    assert launches[0] == launches[2 if own else 1]
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
