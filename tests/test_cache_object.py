"""CompressedCache as an object of its own: made from tensors and lengths, copied, saved and loaded (no GPU)."""
import copy
import io

import numpy as np
import pytest
import torch

from nsa_b200.decode import CompressedCache, _lengths


def _saved(c):
    f = io.BytesIO()
    torch.save(c, f)
    f.seek(0)
    return torch.load(f, weights_only=False)


@pytest.mark.parametrize("how", [lambda c: c, copy.copy, copy.deepcopy, _saved])
def test_cache_from_its_parts(how):
    ck, cv = torch.randn(4, 2, 8), torch.randn(4, 2, 8)
    c = how(CompressedCache(ck, cv, torch.tensor([0, 40, 60, 124, 124]), [0, 1, 1, 4, 4]))
    assert c.cu == [0, 40, 60, 124, 124] and c.cu_c == [0, 1, 1, 4, 4] and c.max_tc == 3
    assert c.cu_dev.tolist() == c.cu and c.cu_c_dev.tolist() == c.cu_c and c.order_dev.tolist() == [2, 0, 1, 3]
    assert c.cu_dev.dtype == torch.int32 and c.order_dev.device == ck.device
    a, b, cu, cu_c = c
    assert torch.equal(a, ck) and torch.equal(b, cv) and cu == c.cu and cu_c == c.cu_c


def test_a_cache_saved_with_its_tables_as_lists_loads():
    """The attributes that a cache had when its tables were lists and tensors."""
    c = CompressedCache.__new__(CompressedCache)
    c.__setstate__(dict(ck=torch.zeros(1, 1, 8), cv=torch.zeros(1, 1, 8), cu=[0, 40], cu_c=[0, 1], cu_dev=None, cu_c_dev=None,
                        order_dev=None, max_tc=1))
    assert c.cu == [0, 40] and c.order_dev.tolist() == [0]


@pytest.mark.parametrize("cu", [[0, 40, 100], (0, 40, 100), np.array([0, 40, 100]), [np.int64(0), np.int32(40), 100.0],
                                torch.tensor([0, 40, 100]), torch.tensor([0.0, 40.0, 100.0]),
                                [torch.tensor(0), torch.tensor(40), torch.tensor(100)]])
def test_lengths_of_any_kind(cu):
    assert list(_lengths(cu)) == [0, 40, 100]


def test_lengths_beyond_32_bits_are_refused():
    with pytest.raises(RuntimeError, match="32 bits"):
        _lengths([0, 2 ** 32 + 40])
