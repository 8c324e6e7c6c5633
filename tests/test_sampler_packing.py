"""The buffer in which a step's sampling parameters go to the device (sampling/sampler.py)."""
import numpy as np
import pytest

from gollmgo_b200 import SamplingParams
from gollmgo_b200.sampling.sampler import pack

PARAMS = [SamplingParams(temperature=0.5 + r, top_k=r, top_p=0.1 * r, seed=(1 << 63) + r) for r in range(4)]


def check(host, R, draws):
    wide = host[:4 * R].view(np.int64)
    assert wide[:R].view(np.uint64).tolist() == [(1 << 63) + r for r in range(R)] and wide[R:].tolist() == draws
    assert host[4 * R:5 * R].tolist() == list(range(R))
    f32 = host[5 * R:].view(np.float32)
    assert f32[:R].tolist() == [0.5 + r for r in range(R)] and np.allclose(f32[R:], [0.1 * r for r in range(R)])


@pytest.mark.parametrize("draws", [[7, 8, 9], (7, 8, 9), iter([7, 8, 9]), np.array([7, 8, 9]), [7, 8, 9, 10]])
def test_rows_get_their_own_parameters(draws):
    check(pack(PARAMS, draws, 3), 3, [7, 8, 9])             # (more parameters, or draws, than rows: those of the rows)


def test_too_few_are_refused():
    with pytest.raises(ValueError):
        pack(PARAMS, [5], 3)                                # one draw index is not every row's
    with pytest.raises(ValueError):
        pack(PARAMS[:2], [1, 2, 3], 3)
