"""Q-criterion at lattice sizes that leave ragged CTAs, single cells across a direction and
several rounds per thread, with and without solid cells: bit for bit against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 1, 3), (1, 5, 7), (3, 2, 1), (31, 9, 1), (32, 8, 1), (33, 31, 5), (129, 64, 40)])
@pytest.mark.parametrize("with_flags", [False, True])
def test_q_criterion_sizes(gpu_engine_cls, oracle_mod, dims, with_flags):
    nx, ny, nz = dims
    n = nx * ny * nz
    rng = np.random.default_rng(n)
    u = [rng.normal(0.0, 0.05, n).astype(np.float32) for _ in range(3)]
    flags = rng.integers(0, 3, n).astype(np.uint8) if with_flags else None
    ref = oracle_mod.q_criterion(nx, ny, nz, 0.37, *u, flags)
    eng = gpu_engine_cls(0)
    got = eng.q_criterion({"nx": nx, "ny": ny, "nz": nz, "ux": u[0], "uy": u[1], "uz": u[2], "flags": flags}, 0.37)
    for k in ("qValues", "omegaMag", "omegaVec"):
        assert np.array_equal(got[k].view(np.uint32), np.asarray(ref[k]).view(np.uint32)), k
    assert got["maxQ"] == ref["maxQ"] and got["maxOmega"] == ref["maxOmega"]
    eng.close()
