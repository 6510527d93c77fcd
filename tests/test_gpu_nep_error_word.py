"""The error word of the NEP kernels holds one code, also where a call meets several errors (the codes are
consecutive numbers), and the evaluation's message names it."""
import numpy as np
import pytest
import torch

from matpl_gb300 import _lib, nep as NP, nep_ops, ops, structures

pytestmark = pytest.mark.gpu
DEV = "cuda"


def t(a, dt=torch.float64):
    return torch.tensor(np.ascontiguousarray(a), dtype=dt, device=DEV)


def case():
    cfg = NP.NepConfig(atom_type=[3, 14])
    fr = NP.frames_from_structures([structures.random_packed(60, 0.05, [3, 14], [0.5, 0.5], seed=1)], 6.0)
    tm = t(np.arange(60) % 2, torch.int64)
    na = t(fr.num_atom.reshape(-1, 1), torch.int64)
    args = [na, tm, torch.arange(2, device=DEV), t(fr.box), t(fr.box_orig), t(fr.num_cell, torch.int64),
            t(fr.position), 6.0, 4.0, 200, 100, True]
    return cfg, args, ops.calculate_neighbor(*args)


def test_bad_type_and_bad_index():
    cfg, args, (a, b, la, lb, ra, rb) = case()
    bad, good, la = args[1].clone(), la, la.clone()
    bad[7] = 9                                     # 2
    la[11, 0] = 60                                 # 5: the first index past the atoms
    m = NP.NEP(cfg, NP.init_params(cfg, 3, energy_shift=-3.0), "float32", device=DEV, check_errors=False)
    m.evaluate(a, la, ra, b, lb, rb, args[0], bad)
    assert int(m.err.item()) == _lib.KERR_BAD_COUNT
    with pytest.raises(_lib.MatplError, match="list index"):
        m.check_errors = True
        m.evaluate(a, la, ra, b, lb, rb, args[0], bad)
    assert int(m.err.item()) == 0
    with pytest.raises(_lib.MatplError, match="type outside"):
        m.evaluate(a, good, ra, b, lb, rb, args[0], bad)


def test_descriptor_operators():
    cfg, args, (a, b, la, lb, ra, rb) = case()
    bad, la = args[1].clone(), la.clone()
    bad[7], la[11, 0] = 9, 60
    prm = NP.init_params(cfg, 3, energy_shift=-3.0)
    nep_ops.set_check_errors(True)
    with pytest.raises(_lib.MatplError, match="error 5"):
        nep_ops.calculateNepFeat(prm["c_param_2"].to(DEV), ra, la, bad, ra.new_empty(0), 6.0, 0)


def test_bad_type_inside_a_shared_run():
    """Two warps share a run of atoms: a bad type alone is reported, not a hand-off that gave up."""
    cfg = NP.NepConfig(atom_type=[3, 14])
    fr = NP.frames_from_structures([structures.random_packed(2433, 0.05, [3, 14], [0.5, 0.5], seed=2)], 6.0)
    tm = t(np.arange(2433) % 2, torch.int64)
    na = t(fr.num_atom.reshape(-1, 1), torch.int64)
    a, b, la, lb, ra, rb = ops.calculate_neighbor(na, tm, torch.arange(2, device=DEV), t(fr.box), t(fr.box_orig),
                                                  t(fr.num_cell, torch.int64), t(fr.position), 6.0, 4.0,
                                                  112, 60, True)
    tm[1200] = 7
    m = NP.NEP(cfg, NP.init_params(cfg, 3, energy_shift=-3.0), "float32", device=DEV, check_errors=False)
    r = m.evaluate(a, la, ra, b, lb, rb, na, tm)
    assert int(m.err.item()) == _lib.KERR_BAD_TYPE and float(r["Ei"][1200]) == 0.0
