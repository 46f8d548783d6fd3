"""Phrase table close to its limit of three quarters: the dictionary fits at the
first attempt (probe runs stay below the limit for small tables), and one that
does not fit is found again in the full-size table."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SLOTS = 1 << 20


@pytest.mark.parametrize("load,retries", [(0.70, 0), (0.745, 0), (0.80, 1)])
def test_load(pkg, load, retries):
    # random bytes: every phrase is distinct, one window in 16 ends one (the count's deviation is 0.001 of the slots)
    n = int(load * SLOTS * 16)
    t = np.random.default_rng(int(load * 1000)).integers(2, 252, size=n).astype(np.uint8)
    with pkg.Storage(0, tuning={"hash_log2_max": 20}) as st:
        got = st.pfp_bwt(t, 5, 16)
        s = st.stats()
        assert abs(s["d"] / SLOTS - load) < 0.005
        assert s["hash_retries"] == retries
        assert np.array_equal(st.unbwt(got, s["primary_index"]), t)
