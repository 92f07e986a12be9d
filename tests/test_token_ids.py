"""Token ids and wanted places on their way to the device (CPU only)."""

import numpy as np
import pytest
import torch

from glm_tpu_b200.runner.lane_runner import _host_ids, _run


@pytest.mark.parametrize("ids", [[], [5], (1, 2, 3), range(7), [True, False, 9], [np.int64(4), np.uint8(7)], np.arange(6), np.arange(4, dtype=np.uint16), [3.0, 2.7],
                                 torch.arange(5), [torch.tensor(8), 9], [-1, 2**31 - 1, -(2**31)], iter([4, 2])])
def test_ids_become_the_tensor_that_torch_makes_of_them(ids):
    ids = list(ids)
    got = _host_ids(iter(ids))
    assert got.dtype == torch.int32 and torch.equal(got, torch.as_tensor(ids, dtype=torch.int32))


@pytest.mark.parametrize("ids", [[2**31], [1, -(2**31) - 1], ["7"], [None]])
def test_what_is_no_id_is_refused(ids):
    with pytest.raises((RuntimeError, TypeError, ValueError, OverflowError)):
        torch.as_tensor(ids, dtype=torch.int32)
    with pytest.raises((RuntimeError, TypeError, ValueError, OverflowError)):
        _host_ids(ids)


@pytest.mark.parametrize("indices,run", [([4], slice(4, 5)), ([0, 1, 2], slice(0, 3)), ([1, 0], None), ([3, 3], None), ([2, 4], None), ([5, 6, 6], None)])
def test_neighbours_in_order_are_a_slice(indices, run):
    assert _run(indices) == run
