"""The precision form's state, whose rows are padded, going in and out through
every door: upload and download (host and device arrays), save and restore.
Row lengths around a block's threads, a group's values and the padding; every
value comes back as it went in, ghosts included."""
import numpy as np
import pytest
import torch

import fall3d_gb300 as F
from fall3d_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [F.PREC_FP32, F.PREC_FP64])
@pytest.mark.parametrize("nx,ny,nz,nc", [(3, 3, 3, 1), (4, 3, 3, 2), (31, 29, 5, 7), (253, 3, 3, 2), (254, 4, 3, 1),
                                         (255, 3, 3, 1), (257, 5, 3, 1), (2045, 3, 3, 1), (2047, 3, 3, 2)])
def test_state_round_trips(prec, nx, ny, nz, nc, tmp_path):
    s = synth.make_scenario("tiny", seed=1, nx=nx, ny=ny, nz=nz, nc=nc, run_h=0.2)
    r = np.random.default_rng(nx)
    c = r.standard_normal((nc, nz + 2, ny + 2, nx + 2)).astype(np.float32).astype(np.float64)
    dry, wet = r.random((nc + 1, ny, nx)), r.random((nc + 1, ny, nx))
    g = F.Context(s, prec)
    g.upload_state(c, dry, wet)
    path = tmp_path / "state.ckpt"
    g.save(path)
    h = F.Context(s, prec)
    h.restore(path)
    second = tmp_path / "again.ckpt"
    h.save(second)
    assert path.read_bytes() == second.read_bytes()
    d = torch.as_tensor(c, device="cuda")
    torch.cuda.synchronize()
    e = F.Context(s, prec)
    e.upload_state(d)
    back = torch.full_like(d, -1.0)
    torch.cuda.synchronize()
    assert e.lib.f3d_download(e.h, back.data_ptr(), None, None, None, None) == 0
    e.sync()
    assert np.array_equal(back.cpu().numpy(), c)
    for x in (g, h):
        f = x.fields()
        assert np.array_equal(f["c"], c)
        assert np.array_equal(f["cdry"], dry) and np.array_equal(f["cwet"], wet)
    for x in (g, h, e):
        x.close()
