"""The IR convolution on each detector's support only: odd detector counts
(column pairs across instances), rectangular grids with gaps between the arcs'
samples, IRs with and without a DC part (differenced input or not), a support
that reaches the last sample.  Bars of test_gpu_operator.py: 1e-5 relative to
the FP64 oracle."""
import numpy as np
import pytest

from oracle import model as M
from pairs import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,D,T,fmin", [
    (64, 64, 37, 2030, 1e5),   # odd D: pairs straddle two instances
    (64, 64, 8, 1500, 0.0),    # DC in the IR: plain input
    (3, 90, 16, 1400, 1e5),    # wide column spacing: empty samples inside the support
    (40, 40, 5, 0, 1e5),       # support ends at the recording's last samples
])
def test_operator_on_the_support(cuda, nx, nz, D, T, fmin):
    import torch
    from msot_gb300 import Discretization, MSOTmodel, Probe
    fov = (-0.006, 0.006, -0.005, 0.005)
    eir = M.gauss_pulse_eir()
    if T == 0:  # the fewest samples that hold every tap
        d = Discretization(fov, (nx, nz))
        far = M.travel_time_indices(M.ArcProbe(n_det=D, radius=0.02, n_samples=4000, eir=eir,
                                               eir_length=eir.size),
                                    M.Grid(nx, nz, fov), 1500.0, 0).max()
        T = int(far + d.dz / (1500.0 / 4e7)) + 2
    op = M.ArcProbe(n_det=D, radius=0.02, n_samples=T, eir=eir, eir_length=eir.size)
    om = M.Model(op, M.Grid(nx, nz, fov), c=1500.0, fmin=fmin, fmax=12e6, norm=2e-5)
    pm = MSOTmodel(Probe(n_det=D, radius=0.02, n_samples=T, eir=eir, eir_length=eir.size),
                   Discretization(fov, (nx, nz)), 1500.0, False, True, 0, fmin, 12e6, 2e-5,
                   max_batch=3)
    rng = np.random.default_rng(nx)
    x = rng.random((3, nx, nz))
    y = pm.forward(torch.tensor(x, dtype=torch.float32)).cpu().numpy()
    assert rel(y, om.forward(x)) < 1e-5
    s = rng.standard_normal((3, D, T))
    xa = pm.transpose(torch.tensor(s, dtype=torch.float32)).cpu().numpy()
    assert rel(xa, om.transpose(s)) < 1e-5
