"""The four-step transforms of the lengths outside the tuned list (transforms3.cu) against the numpy oracle:
y_to_x, dft_x_realspace and x_to_y for every such length, as the x and as the z length, with kx counts
that are no multiple of a block's lines, in both precisions (FP64 2e-14 relative, FP32 transforms 1e-6)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from channel_passive_b200 import Channel, Config
from oracle import kmm as okmm
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu

LENGTHS = [27, 30, 45, 54, 60, 75, 81, 90, 108, 120, 135, 150, 162, 180, 216, 225, 240, 243, 270, 300, 324, 360,
           375, 432, 480]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("i", range(len(LENGTHS)))
def test_transforms_match_oracle(i, precision):
    nx, nz, ny = LENGTHS[i] * 2 // 3, LENGTHS[(7 * i + 3) % len(LENGTHS)] * 2 // 3, 19
    nxh, nx32, nz32 = nx // 2, nx * 3 // 2, nz * 3 // 2
    tol = 1e-6 if precision else 2e-14
    rng = np.random.default_rng(i)
    U = rng.standard_normal((4, nz, nxh, ny)) + 1j * rng.standard_normal((4, nz, nxh, ny))
    line = torch.float32 if precision else torch.float64
    X = torch.zeros((10, ny, nz32, nxh, 2), dtype=line, device="cuda")
    ref = np.zeros((10, ny, nz32, nxh), dtype=np.complex128)
    cfg = Config(nx=nx, ny=ny, nz=nz, precision=precision, fixed_dt=1)
    as_complex = lambda t: torch.view_as_complex(t.double().contiguous()).cpu().numpy()
    with Channel(cfg) as ch:
        dev = torch.from_numpy(U).cuda()
        for k, f in enumerate((0, 1, 2, 6)):
            ch.y_to_x(dev[k], X[f])
            ref[f] = okmm.y_to_x(U[k], nz32)
        torch.cuda.synchronize()
        for f in (0, 1, 2, 6):
            assert rel_l2(as_complex(X[f]), ref[f]) < tol, ("y_to_x", f)
        if not precision:
            X = torch.view_as_real(torch.from_numpy(ref)).cuda().contiguous()
        else:
            ref = np.stack([as_complex(X[f]) for f in range(10)])
        dxr, dzr = nx / (2 * np.pi * cfg.lmfx), nz / (2 * np.pi * cfg.lmfz)
        dyr = okmm.dyr_vector(ch.y, 1.0)
        velmax = torch.zeros(1, dtype=torch.float64, device="cuda")
        ch.dft_x_realspace(X, 1, velmax)
        torch.cuda.synchronize()
        vm = okmm.dft_x_realspace(ref, nx, 1, dxr, dzr, dyr)
        assert abs(float(velmax) - vm) <= 10 * tol * vm
        for f in (0, 1, 2, 3, 4, 6, 7, 8):
            assert rel_l2(as_complex(X[f]), ref[f]) < 2 * tol, ("x", f)
        out = torch.zeros((nz, nxh, ny), dtype=torch.complex128, device="cuda")
        for f in (1, 7):
            src = as_complex(X[f])
            ch.x_to_y(X[f], out, rescale=False)
            torch.cuda.synchronize()
            assert rel_l2(out.cpu().numpy(), okmm.x_to_y(src, nz)) < tol, ("x_to_y", f)
