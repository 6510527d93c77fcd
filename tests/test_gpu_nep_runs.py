"""FP32 NEP evaluation where the run of atoms is shared by two warps (lists too wide for two
8-run blocks per SM) and where it is not, around the sizes at which runs grow to 2 and 3 atoms,
with frame boundaries inside runs and an atom of a bad type: against the FP64 evaluation of the
same lists (forces to 1e-4 eV/A, the form's bar; energies and virial to 1e-5 of their size per
atom), and both list widths against each other."""
import numpy as np
import pytest
import torch

from matpl_gb300 import _lib, nep as NP, ops, structures

pytestmark = pytest.mark.gpu
DEV = "cuda"


def t(a, dt=torch.float64):
    return torch.tensor(np.ascontiguousarray(a), dtype=dt, device=DEV)


@pytest.mark.parametrize("counts", [(1217,), (608, 1, 700, 1200), (2433,), (1216 * 2 + 1, 37)])
def test_paired_runs_match_fp64(counts):
    cfg = NP.NepConfig(atom_type=[3, 14])
    sts = [structures.random_packed(n, 0.05 if n > 300 else 0.01, [3, 14], [0.5, 0.5], seed=n) for n in counts]
    fr = NP.frames_from_structures(sts, 6.0)
    rng = np.random.default_rng(len(counts))
    tm = t(rng.integers(0, 2, fr.natoms), torch.int64)
    na = t(fr.num_atom.reshape(-1, 1), torch.int64)
    prm = NP.init_params(cfg, 3, energy_shift=-3.0)
    prm["q_scaler"] = torch.full((cfg.feature_nums,), 0.1, dtype=torch.float64)
    args = (na, tm, torch.arange(2, device=DEV), t(fr.box), t(fr.box_orig),
            t(fr.num_cell, torch.int64), t(fr.position), 6.0, 4.0)
    out = {}
    for width in ((72, 28), (112, 60)):          # two 8-warp blocks per SM / one paired block
        a, b, la, lb, ra, rb = ops.calculate_neighbor(*args, *width, True)
        for prec in ("float32", "float64"):
            m = NP.NEP(cfg, prm, prec, device=DEV)
            r = m.evaluate(a, la, ra, b, lb, rb, na, tm)
            out[(width[0], prec)] = {k: v.double() for k, v in r.items()}
    for w in (72, 112):
        g, e = out[(w, "float32")], out[(112, "float64")]
        assert float((g["Force"] - e["Force"]).abs().max()) <= 1e-4
        assert float(((g["Etot"] - e["Etot"]).abs() / na.flatten()).max()) <= 1e-5 * 5
        assert float(((g["Virial"] - e["Virial"]).abs() / na).max()) <= 1e-5 * 10
    assert torch.equal(out[(72, "float32")]["Ei"], out[(112, "float32")]["Ei"])
    # an atom of a bad type in the middle of a run: flagged, its energy 0, the others untouched
    bad = tm.clone()
    bad[fr.natoms // 2] = 7
    m = NP.NEP(cfg, prm, "float32", device=DEV, check_errors=False)
    r = m.evaluate(a, la, ra, b, lb, rb, na, bad)
    assert int(m.err.item()) & _lib.KERR_BAD_TYPE and float(r["Ei"][fr.natoms // 2]) == 0.0
    assert bool(torch.isfinite(r["Force"]).all())
