"""Sphere placement around the 32 configurations a warp lays out at a time and
the 64 of a block, into 16-byte aligned and unaligned outputs: bit-identical to
the oracle's FP32 mirror with the device's __sinf/__cosf values replayed, and
nothing written past the last configuration."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 1000])
@pytest.mark.parametrize("detailed", [False, True])
@pytest.mark.parametrize("offset", [0, 1])
def test_fk_spheres_sizes(cuda, pkg, orc, n, detailed, offset):
    W = pkg.workloads
    q = W.random_configs(np.random.default_rng(n), n, 1)
    dq = cuda.from_numpy(q).cuda()
    c, s = pkg.debug_trig(dq.reshape(-1))
    spheres = 59 if detailed else 11
    buf = cuda.full((n * spheres * 3 + 8,), 7.5, dtype=cuda.float32, device="cuda")
    bases = W.bases_config2()
    robots = pkg.RobotSet(4, bases)
    lib = pkg.library()
    stream = cuda.cuda.current_stream().cuda_stream
    assert lib.mrpop_fk_spheres(robots.handle, 2, dq.data_ptr(), n, int(detailed), buf.data_ptr() + 4 * offset,
                                stream) == 0
    cuda.cuda.synchronize()
    trig = orc.TrigTable(q.ravel(), c.cpu().numpy(), s.cpu().numpy())
    ref = orc.fk_spheres(bases[2], q, detailed, fp64=False, trig=trig).astype(np.float32)
    got = buf.cpu().numpy()
    end = offset + n * spheres * 3
    assert np.array_equal(got[offset:end].reshape(n, spheres, 3), ref)
    assert (got[:offset] == 7.5).all() and (got[end:] == 7.5).all()
