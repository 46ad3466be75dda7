"""FemPack's host side without a device: the buffer that joins the models' states."""
import numpy as np

from artisynth_core_b200.femmodel import FemPack


def test_join_buffer_is_reused_and_given_back():
    p = FemPack([])
    a, b = np.arange(6.0).reshape(2, 3), -np.arange(9.0).reshape(3, 3)
    one = p._joined(0, [a, b])
    assert np.array_equal(one, np.concatenate([a, b]).reshape(-1))
    assert np.shares_memory(one, p._joined(0, [b, a]))
    assert np.array_equal(p._joined(1, [a, b]), np.concatenate([a, b]).reshape(-1))
    assert not np.shares_memory(p._joined(0, [a]), p._joined(1, [a]))
    p.close()
    assert not any(isinstance(v, list) and any(isinstance(x, np.ndarray) for x in v) for v in vars(p).values())
    assert np.array_equal(p._joined(0, [b]), b.reshape(-1))
