"""Flat windows without a flat neighbour: settled at candidate compaction (r^2 <= 2m),
left to the refine above that.  Counts and values against the FP64 profile; the values
of such windows are 2m exactly."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dist,rows", [("fp32", 0), ("fp16", 0), ("fp16", 64)])
# series length, m, first value and length of the flat run: a short series whose middle
# windows have no neighbour at all, runs at either end, more flat windows than one tile
@pytest.mark.parametrize("n,m,at,run", [(260, 128, 60, 140), (20000, 40, 0, 45), (20000, 40, 19000, 1000),
                                        (40000, 120, 9000, 238)])
def test_flat_windows_without_flat_neighbour(dist, rows, n, m, at, run):
    import torch

    import paddi_b200 as P
    x = np.cumsum(np.random.default_rng(5).standard_normal(n)).astype(np.float32)
    x[at:at + run] = x[at]
    nn, _ = O.nn_profile(x, m)
    N = n - m + 1
    k = {"fp32": P.DIST_FP32, "fp16": P.DIST_SPLIT_FP16}[dist]
    dx = torch.from_numpy(x).cuda()
    fl = torch.empty(N, dtype=torch.int32, device="cuda")
    q = torch.empty(N, dtype=torch.float32, device="cuda")
    with P.Context(device=0, distance_kernel=k, tile_rows=rows) as ctx:
        for r2 in (1.0, 1.5 * m, np.nextafter(np.float32(2 * m), np.float32(0)), 2.0 * m,
                   2.0 * m + 1.0):
            got = ctx.do_pd3(dx.data_ptr(), n, m, float(r2), fl.data_ptr(), q.data_ptr(),
                             torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            want = nn.astype(np.float32) >= np.float32(r2)
            has = np.isfinite(nn) & (nn < 1e30)  # windows with a neighbour
            f = fl.cpu().numpy().astype(bool)
            assert np.array_equal(f[has], want[has]), r2
            assert got == f.sum()
            exact = has & want & (nn == 2.0 * m)
            assert (q.cpu().numpy()[exact] == np.float32(2 * m)).all(), r2
