"""NEP neighbor lists at the edges of the FP32 tests and the shortened exact arithmetic, bit for bit
against the oracle: replicated and single small cells whose half thickness is the cutoff (pairs
at the fold's tie), sheared cells, more frames than a warp has lanes (empty-ish ones among them),
atoms on the coordinate planes (zero components, whole cells apart) and unwrapped positions."""
import numpy as np
import pytest
import torch

from matpl_gb300 import nep as NP, ops
from oracle import nep_oracle as NO

pytestmark = pytest.mark.gpu
DEV = "cuda"
RC, RA = 6.0, 4.0


def frames(cells):
    """cells: [(lattice rows, cartesian positions)]"""
    ex = [NP.expand_box(np.asarray(lat, dtype=np.float64), RC) for lat, _ in cells]
    return NP.NepFrames(np.concatenate([p for _, p in cells]),
                        np.zeros(sum(len(p) for _, p in cells), dtype=np.int64),
                        np.array([len(p) for _, p in cells], dtype=np.int64),
                        np.stack([e[0] for e in ex]), np.stack([e[1] for e in ex]),
                        np.stack([e[2] for e in ex]))


def check(fr, mr=200, ma=100):
    want = NO.neighbor(fr, RC, RA, mr, ma)
    t = lambda a, dt=torch.float64: torch.tensor(np.ascontiguousarray(a), dtype=dt, device=DEV)  # noqa: E731
    got = ops.calculate_neighbor(t(fr.num_atom, torch.int64), t(fr.type_map, torch.int64),
                                 torch.zeros(1, dtype=torch.int64, device=DEV), t(fr.box), t(fr.box_orig),
                                 t(fr.num_cell, torch.int64), t(fr.position), RC, RA, mr, ma, True)
    NN_r, NN_a, NL_r, NL_a, Ri_r, Ri_a = (x.cpu().numpy() for x in got)
    assert np.array_equal(NN_r, want[0]) and np.array_equal(NN_a, want[1])
    for n, NL, R, NLo, Ro in ((NN_r, NL_r, Ri_r, want[2], want[4]), (NN_a, NL_a, Ri_a, want[3], want[5])):
        occ = np.arange(NL.shape[1])[None] < n[:, None]
        assert np.array_equal(NL[occ], NLo[occ])
        assert np.array_equal(R[occ].view(np.uint64), Ro[occ].view(np.uint64))
        assert (NL[~occ] == -1).all() and (R[~occ] == 0).all()
    assert NN_r.sum() > 0


@pytest.mark.parametrize("L", [12.0, 12.0000001, 11.9999999, 6.0, 3.1])
@pytest.mark.parametrize("shear", [0.0, 0.25, 0.5])
def test_ties_of_the_fold(L, shear):
    lat = np.eye(3) * L
    lat[1, 0] = shear * L
    lat[2, 1] = -0.5 * shear * L
    n = max(1, int(round(L / 3)))
    g = np.stack(np.meshgrid(*(np.arange(n),) * 3, indexing="ij"), -1).reshape(-1, 3) / n
    rng = np.random.default_rng(int(L * 10))
    check(frames([(lat, g @ lat), (lat, (g + 1e-9 * rng.normal(size=g.shape)) @ lat)]))


def test_far_apart_and_needle_cells():
    rng = np.random.default_rng(9)
    lat = np.eye(3) * 7.0
    far = rng.uniform(0, 7, (9, 3)) + 7.0 * rng.integers(-20000, 20000, (9, 3))
    needle = np.diag([6.5, 6.5, 6.5])
    needle[1] += 9 * needle[0]
    needle[2] += 7 * needle[1]
    check(frames([(lat, far), (needle, rng.uniform(0, 1, (12, 3)) @ needle)]), 400, 200)


def test_many_frames():
    rng = np.random.default_rng(5)
    cells = []
    for k in range(70):
        lat = np.diag(rng.uniform(4, 14, 3)) + (rng.normal(0, 0.6, (3, 3)) if k % 3 else 0.0)
        n = 1 + (k * 7) % 19
        cells.append((lat, rng.uniform(-1.5, 2.5, (n, 3)) @ lat))
    check(frames(cells))


@pytest.mark.parametrize("shift", [0.0, 0.5, -37.0])
def test_large_cell_zero_components(shift):
    n, a = 9, 3.0
    g = np.stack(np.meshgrid(*(np.arange(n),) * 3, indexing="ij"), -1).reshape(-1, 3) * a
    g = g + np.where(np.arange(len(g))[:, None] % 5 == 0, shift * n * a, 0.0)     # unwrapped
    jit = g + np.random.default_rng(1).normal(0, 0.2, g.shape)
    check(frames([(np.eye(3) * n * a, g), (np.eye(3) * n * a, jit), (np.eye(3) * n * a, -g)]))
