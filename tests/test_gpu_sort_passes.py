"""The radix sort's skipped passes (thrust::sort_by_key's role, engine.cu:98-99):
keys that vary in no digit, in one, in the outer two, in the middle two, in
all, at sizes around a tile and a CTA's share, with and without allocation."""
import numpy as np
import pytest

from parity import morton_reference, stable_sort_reference

pytestmark = pytest.mark.gpu

# Coordinate bit k is key bits 3k..3k+2: digit 0 = coordinate bits 0..2 (in
# part), digit 1 = 3..5, digit 2 = 5..7, digit 3 = 8, 9.
KINDS = {
    "equal": [0],
    "digit0": [0, 1, 2, 3],
    "digit3": [0, 256, 512, 768],
    "digits0_3": [0, 1, 512, 513],
    "digits1_2": [0, 8, 64, 72],
    "all": list(range(0, 1024, 7)),
}


@pytest.mark.parametrize("n", [1, 33, 2047, 2049, 40_000])
@pytest.mark.parametrize("static", [False, True])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_sort_passes(gpu_ok, mpm, kind, n, static):
    import torch
    rng = np.random.default_rng(n)
    pos = (rng.choice(KINDS[kind], (3, n)) + 0.9 * rng.random((3, n))).astype(np.float32)
    d = torch.from_numpy(pos).cuda()
    keys = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    perm = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    sort = mpm.sort_particles_device_static if static else mpm.sort_particles_device
    for _ in range(2):  # the second call finds what the first left in the scratch
        sort(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), n, keys.data_ptr(), perm.data_ptr(),
             torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    want = morton_reference(pos)
    assert np.array_equal(keys.cpu().numpy(), want)
    assert np.array_equal(perm.cpu().numpy(), stable_sort_reference(want))
