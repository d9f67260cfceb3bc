"""The sort's group path and its way to the full radix sort, against a stable
numpy sort: sizes at the edges of one group, of one and two top digits, keys
that overfill a group or a finer range, keys with bits above the fingerprints'
59, a large sort after a small one on the same scratch."""
import numpy as np
import pytest
import torch

import empanada_b200
from test_gpu_sort import _expected, _keys

pytestmark = pytest.mark.gpu


def _check(sort, keys, vals):
    dk = torch.from_numpy(keys.view(np.int64).copy()).cuda()
    dv = torch.from_numpy(vals.view(np.int32).copy()).cuda()
    torch.cuda.synchronize()
    sort(dk.data_ptr(), dv.data_ptr(), len(keys))
    ek, ev = _expected(keys, vals)
    assert (dk.cpu().numpy().view(np.uint64) == ek).all()
    assert (dv.cpu().numpy().view(np.uint32) == ev).all()


def _vals(rng, n):
    return rng.integers(0, 2**32, size=n, dtype=np.uint64).astype(np.uint32)


SIZES = [2, 33, 2900, 2901, 4096, 4097, 5801, 256 * 2900, 256 * 2900 + 1, 1_000_003, 2_500_001]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("copies", [1, 3, 40, 700])
def test_sizes_and_equal_keys(engine, n, copies):
    rng = np.random.default_rng(n + copies)
    keys = _keys(rng, n, max(1, n // copies))
    vals = _vals(rng, n)
    _check(engine.sort_pairs, keys, vals)
    if n <= empanada_b200.SORT_STATIC_MAX_PAIRS:
        _check(empanada_b200.sort_pairs_static, keys, vals)


KINDS = {
    "one_key": lambda r, n: np.full(n, 7 << 32 | 9, np.uint64),
    "low_half": lambda r, n: _keys(r, n, n) >> np.uint64(1) & ~np.uint64(7 << 29),
    "narrow": lambda r, n: (np.uint64(123456) << np.uint64(32)) | r.integers(0, 536870879, n, dtype=np.uint64),
    "few_keys": lambda r, n: _keys(r, n, 5),
    "any_bits": lambda r, n: r.integers(0, 1 << 62, n, dtype=np.uint64) * np.uint64(4) + r.integers(0, 4, n).astype(np.uint64),
    "one_high_key": lambda r, n: np.where(np.arange(n) == n // 3, np.uint64(1 << 61), _keys(r, n, n)),
    "in_order": lambda r, n: np.sort(_keys(r, n, n)),
    "reversed": lambda r, n: np.sort(_keys(r, n, n))[::-1].copy(),
}


@pytest.mark.parametrize("kind", sorted(KINDS))
@pytest.mark.parametrize("n", [100, 4096, 50_000, 900_001])
def test_uneven_keys(engine, kind, n):
    rng = np.random.default_rng(n)
    keys = KINDS[kind](rng, n).astype(np.uint64)
    vals = _vals(rng, n)
    _check(engine.sort_pairs, keys, vals)
    _check(empanada_b200.sort_pairs_static, keys, vals)


def test_sizes_in_turn_on_one_scratch():
    """Bounds of a smaller sort lie where a larger one has look-back words."""
    rng = np.random.default_rng(1)
    with empanada_b200.Engine(0) as eng:
        for n in [2_000_000, 5000, 1_999_999, 800_000, 4097, 2_000_000, 100_000]:
            _check(eng.sort_pairs, _keys(rng, n, n), _vals(rng, n))
            _check(eng.sort_pairs, _keys(rng, n, 3), _vals(rng, n))
