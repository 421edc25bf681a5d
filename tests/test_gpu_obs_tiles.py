"""Push-T observations at the edges of the kernel's tiles, byte for byte
against the oracle: the smallest images, odd row lengths, environments of one
and of many tiles, windows that the shapes leave or fill, an empty window, and
an output at an odd address."""
import numpy as np
import pytest

from avbd_b200 import demos
from avbd_b200.solver import GPUSolver

pytestmark = pytest.mark.gpu


def _pair(oracle_lib, envs=5):
    s, e = demos.pusht_scene(envs, seed=7)
    g, o = GPUSolver(s), oracle_lib.OracleSolver(s, threads=2)
    g.step(3)
    assert o.step(3) == 0
    return g, o, demos.pusht_env_table(e)


@pytest.mark.parametrize("res", [2, 3, 33, 73, 74, 130, 1025])
def test_obs_bytes_at_tile_edges(cuda_lib, oracle_lib, res):
    g, o, table = _pair(oracle_lib, 5 if res < 1000 else 2)
    for half in (3.25, 0.2, -3.25, 0.0):
        for t in table:
            t.goal[1] = half
        a, b = g.render_pusht_obs(table, res), o.render_pusht_obs(table, res)
        assert np.array_equal(a, b), (half, int((a != b).any(-1).sum()))


def test_obs_at_an_odd_address(cuda_lib, oracle_lib):
    import torch
    g, o, table = _pair(oracle_lib)
    res = 51
    n = 5 * res * res * 3
    for shift in (0, 1, 7, 15):
        buf = torch.full((n + 64,), 77, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        g.render_pusht_obs(table, res, device_out=buf.data_ptr() + 16 + shift)
        g.synchronize()
        host = buf.cpu().numpy()
        assert np.array_equal(host[16 + shift:16 + shift + n].reshape(5, res, res, 3), o.render_pusht_obs(table, res))
        assert (host[:16 + shift] == 77).all() and (host[16 + shift + n:] == 77).all()
