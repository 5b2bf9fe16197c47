"""CPU model of the pencil grid of the box passes whose columns are moved in
pairs of cells (gf_smooth.cu, box_geom<AXIS, true> and smooth_reg_box_kernel):
every column of the box is filtered by exactly one pair, both cells of a pair lie
in one row of the mesh at an even offset, and a column beside the box is never
stored."""
import numpy as np
import pytest

P = 32  # pencils per tile


def _pair_lo(lo):
    return lo & ~1


def _pair_len(lo, hi):
    return 0 if hi < lo else (hi | 1) - (lo & ~1) + 1


@pytest.mark.parametrize("nx", [64, 128, 256])
def test_every_column_once(nx):
    rng = np.random.default_rng(nx)
    mx = 2 * (nx // 2 + 1)
    boxes = [(0, nx - 1, 3), (0, 0, 1), (nx - 1, nx - 1, 5), (1, 2, 7), (1, 1, 40), (31, 32, 2), (5, 4, 3)]
    boxes += [(*sorted(rng.integers(0, nx, 2)), int(rng.integers(1, 50))) for _ in range(60)]
    for a0, a1, nv in boxes:
        u0, nu = _pair_lo(int(a0)), _pair_len(int(a0), int(a1))
        assert nu % 2 == 0 and u0 % 2 == 0 and u0 + nu <= mx
        done = np.zeros((nv, mx), int)
        for t in range((nu * nv + P - 1) // P):
            f0 = t * P
            npen = min(P, nu * nv - f0)
            assert npen % 2 == 0
            for c in range(npen // 2):
                v, u = divmod(f0 + 2 * c, nu)
                x = u0 + u
                assert x % 2 == 0 and u + 1 < nu and x + 1 < mx  # one row, 8-byte aligned
                if x >= a0:
                    done[v, x] += 1
                if x + 1 <= a1:
                    done[v, x + 1] += 1
        want = np.zeros_like(done)
        if a1 >= a0:
            want[:, a0:a1 + 1] = 1
        assert np.array_equal(done, want)
