"""A planned batch's descriptor arrays keep their shapes and types on the device, each on a boundary of its own, although they
arrive in one copy: a caller may write new positions or k-points into them."""
import numpy as np
import torch

from slakonet_gb300 import engine as E
from test_groups_host import _batch


def test_arrays_keep_shape_type_and_values():
    db = _batch((1, 4, 9), nk=3)
    p = db.plan
    for t, a, dtype in ((db.pos, p.positions, torch.float64), (db.cells, p.cells, torch.float64),
                        (db.rng, p.image_range, torch.int32), (db.kp, p.kpoints, torch.float64),
                        (db.atom_ptr, p.atom_ptr, torch.int32), (db.hs_off, p.hs_off, torch.int64)):
        assert tuple(t.shape) == a.shape and t.dtype == dtype and np.array_equal(t.numpy(), a)
        assert t.is_contiguous() and t.data_ptr() % 16 == 0
    db.pos.copy_(torch.as_tensor(p.positions + 0.5))
    assert np.array_equal(db.pos.numpy(), p.positions + 0.5) and np.array_equal(db.cells.numpy(), p.cells)


def test_every_type_and_empty_arrays_in_one_copy():
    arrays = [(np.zeros((0, 3)), np.float64), (np.arange(5), np.int32), (np.zeros(0), np.int64),
              (np.arange(6.0).reshape(2, 3)[:, ::-1], np.float64), (np.array([2 ** 40]), np.int64)]
    got = E._to_device(arrays, torch.device("cpu"))
    for (a, t), v in zip(arrays, got):
        assert tuple(v.shape) == (a.size,) and np.array_equal(v.numpy(), a.astype(t).reshape(-1))
