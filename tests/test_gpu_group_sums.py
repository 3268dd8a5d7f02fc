"""Grouped FP64 sums of whole numbers: every thread's part has 48 bits and the sum 53, so the answer is
exact, whatever the order of the additions, if a block sums its threads' parts no worse than doubles do."""
import numpy as np
import pytest

from widequery import GROUPS, wide_groupby_query, wide_table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncol", [1, 2, 3])
@pytest.mark.parametrize("n", [1, 31, 33, 511, 513, 2047, 4096, 4097, 7999])
def test_whole_number_sums_of_53_bits_are_exact(eng, n, ncol):
    # at most 4096 rows a block, so 8 rows and 2^45 a thread; at most 2^55 / 4 in a group
    t = wide_table(n, ncol, seed=n)
    rng = np.random.default_rng(n + ncol)
    vals = [rng.integers(1, 2**42, n) for _ in range(ncol)]
    for c, v in zip(t.columns[3:], vals):
        c.data[:] = v.astype(np.float64)
    got = eng.compile(wide_groupby_query(t.get_data_type(), ncol)).run(eng.upload(t))
    ka, kb = t.columns[1].data, t.columns[2].data
    for (a, b), sums in zip(GROUPS, got):
        m = (ka == a) & (kb == b)
        sums = sums if isinstance(sums, tuple) else (sums,)
        for v, s in zip(vals, sums):
            assert int(v[m].sum()) < 2**53
            assert int(s) == int(v[m].sum())
