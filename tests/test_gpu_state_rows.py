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


@pytest.mark.parametrize("nx", [12, 13, 14, 31])
def test_steps_after_a_restore(nx, tmp_path):
    """A restore uses the step's second buffer: the steps that follow in the
    same context give the bits of those that followed the save, whatever the
    padding and whichever buffer the state was in."""
    s = synth.make_scenario("small", seed=6, nx=nx, ny=11, nz=9, nc=3, run_h=0.5)
    g = F.Context(s, F.PREC_FP32)
    g.meteo(0)
    g.source(0)
    for before in (2, 3):
        g.step(before)
        t = g.state()
        path = tmp_path / f"{before}.ckpt"
        g.save(path)
        g.step(5)
        want, out = g.fields(), g.state()["outmass"]
        g.restore(path)
        g.meteo(0)
        g.source(0)
        g.set_time(t["time"], t["iiter"])
        g.step(5)
        got = g.fields()
        for k in ("c", "cdry", "cwet"):
            assert np.array_equal(got[k], want[k]), (before, k)
        assert g.state()["outmass"] == out
    g.close()
