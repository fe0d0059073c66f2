"""Calls with less workspace than they would like.

The limit of pEVSL_B200_SetWorkspaceLimit refuses larger workspaces as a full
GPU would, without filling one.
"""
import numpy as np
import pytest

import pevsl_b200 as pv
from pevsl_b200.problems import laplacian

pytestmark = pytest.mark.gpu


@pytest.fixture
def limit():
    lib = pv.load()
    lib.pEVSL_B200_ReleaseWorkspace()
    yield lib.pEVSL_B200_SetWorkspaceLimit
    lib.pEVSL_B200_SetWorkspaceLimit(0)
    lib.pEVSL_B200_ReleaseWorkspace()
    lib.pEVSL_B200_LastError()


@pytest.mark.parametrize("bases", [1, 2, 5])
def test_lanczos_dos_takes_fewer_runs_at_a_time(gpu, limit, bases):
    """The same bits with memory for one, two or five bases, and an error
    with less than one."""
    M = pv.Matrix.from_csr(*laplacian(30, 31, 29))
    nvec, msteps = 11, 25
    one = 8 * ((M.n + 31) // 32 * 32) * (msteps + 1)
    outs = []
    with pv.Instance(M) as ev:
        for bytes_ in (0, int((bases + 0.5) * one)):
            ev.lib.pEVSL_B200_ReleaseWorkspace()
            limit(bytes_)
            pv.set_rng(pv.RNG_GAUSS, 11)
            outs.append(ev.landos(nvec, msteps, 61, [0.5, 6.0, 0.0, 12.0]))
        ev.lib.pEVSL_B200_ReleaseWorkspace()
        limit(one // 2)
        assert ev.landos(nvec, msteps, 61, [0.5, 6.0, 0.0, 12.0])[0] == pv.ERR_NOMEM
    M.free()
    assert outs[0][0] == outs[1][0] == 0
    assert np.array_equal(outs[0][2], outs[1][2]) and outs[0][3] == outs[1][3]


@pytest.mark.parametrize("mdeg", [1, 127, 128, 129, 4000])
def test_kpm_workspace_does_not_grow_with_the_moments(gpu, limit, mdeg):
    """64 vectors at 205 blocks: 210 KB of partial sums per step, 420 MB for
    all steps of 4000 moments; 32 MB do for any number."""
    M = pv.Matrix.from_csr(*laplacian(41, 40, 1))
    outs = []
    with pv.Instance(M) as ev:
        for bytes_ in (0, 32 << 20):
            ev.lib.pEVSL_B200_ReleaseWorkspace()
            limit(bytes_)
            pv.set_rng(pv.RNG_GAUSS, 5)
            outs.append(ev.kpmdos(mdeg, 1, 64, [0.5, 6.0, 0.0, 8.0]))
    M.free()
    assert outs[0][0] == outs[1][0] == 0
    assert np.array_equal(outs[0][1], outs[1][1]) and outs[0][2] == outs[1][2]


def test_the_tuner_gives_its_scratch_back(gpu):
    """The first product with a general matrix times the kernels' forms on
    scratch vectors of 256 MB here; afterwards the device has them back, but
    for at most 64 MB and the matrix's own offsets (80 MB)."""
    import torch
    n = 8_000_000
    rng = np.random.default_rng(0)
    cols = np.arange(n, dtype=np.int64)[:, None] + np.array([-40, -3, 0, 3, 40])
    ok = (cols >= 0) & (cols < n)
    ia = np.concatenate([[0], np.cumsum(ok.sum(1))]).astype(np.int32)
    M = pv.Matrix.from_csr(n, ia, cols[ok].astype(np.int32), rng.standard_normal(int(ia[-1])))
    x, y = pv.Vector(n, np.ones(n)), pv.Vector(n)
    lib = pv.load()
    assert lib.pEVSL_B200_Sync() == 0
    before = torch.cuda.mem_get_info()[0]
    lib.pEVSL_ParcsrMatvec(M.A, x.pv, y.pv)
    assert lib.pEVSL_B200_Sync() == 0
    after = torch.cuda.mem_get_info()[0]
    M.free()
    assert before - after < 200 << 20
