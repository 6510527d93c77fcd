"""A DP model copied or pickled as a whole starts without a kept type map, also one whose pickle holds the
earlier cache instead."""
import copy
import io
import pickle

import numpy as np
import torch

from matpl_gb300 import dp, params as P


def test_copies_and_pickles():
    cfg = P.DPConfig(atom_type=[3, 14], maxNeighborNum=20)
    stats = np.zeros((2, 2 * 20 * 4)), np.ones((2, 2 * 20 * 4))
    m = dp.DP(cfg, P.init_params(cfg, 5), *stats, device="cpu")
    m._order._entry = ("key", torch.zeros(3), None)
    m._order._answers[1] = (torch.zeros(1), None)
    old = copy.deepcopy(m)
    del old.__dict__["_order"]
    old._perm_cache = {}
    for c in (copy.deepcopy(m), pickle.loads(pickle.dumps(m)), pickle.loads(pickle.dumps(old))):
        assert c._order._entry is None and c._order._answers == {} and c._order is not m._order
        assert torch.equal(c.packed, m.packed)
    torch.save(m, io.BytesIO())
