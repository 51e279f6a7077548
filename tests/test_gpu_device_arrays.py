"""Particle arrays on the scene's device are read and written in place (others go through the staging buffer): the same
values either way, at counts around a warp's and a block's, in the caller's order after a substep's sort."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

fe = pytest.importorskip("fluide_engine_b200")
torch = pytest.importorskip("torch")
from fluide_engine_b200._abi import check, ptr  # noqa: E402


@pytest.mark.parametrize("solver", [fe.FLIP, fe.APIC])
@pytest.mark.parametrize("count", [1, 31, 32, 33, 255, 256, 257, 1000])
def test_device_and_host_arrays_agree(solver, count):
    rng = np.random.default_rng(count)
    host = [rng.uniform(0.1, 0.9, (count, 3)), rng.standard_normal((count, 3)), rng.standard_normal((count, 9))]
    host = [a.astype(np.float32) for a in host]
    dev = [torch.from_numpy(a).cuda() for a in host]
    torch.cuda.synchronize()
    got = []
    for arrays in (host, dev):
        s = fe.Scene((12, 10, 9), solver=solver, max_cfl=1.0)
        s.set_particles(*arrays)
        s.run_stages(1 / 240, fe.STAGE_SORT, fe.STAGE_SORT)  # the slots are permuted, the particles are not changed
        out = [torch.full_like(a, -7.0) for a in dev]
        torch.cuda.synchronize()
        check(fe.lib().fe_scene_get_particles(s.handle, ptr(out[0]), ptr(out[1]), ptr(out[2]), count))
        want = host if solver == fe.APIC else host[:2] + [np.zeros_like(host[2])]
        for a, b, c in zip(out, s.particles(), want):
            assert np.array_equal(a.cpu().numpy(), b) and np.array_equal(b, c)
        mixed = torch.full_like(dev[1], -7.0)  # one destination here, one on the host, one not asked for
        pos = np.zeros_like(host[0])
        torch.cuda.synchronize()
        check(fe.lib().fe_scene_get_particles(s.handle, ptr(pos), ptr(mixed), None, count))
        assert np.array_equal(pos, host[0]) and np.array_equal(mixed.cpu().numpy(), host[1])
        s.close()
