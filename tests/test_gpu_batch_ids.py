"""A batch's ids share one space of at most 2^31 - 2: larger ones are refused,
the largest 32-bit id (whose successor wraps to 0) among them, by every form a
group is counted in."""
import numpy as np
import pytest

import oracle
import signed_triangle_counting_b200 as stc
from signed_triangle_counting_b200 import _capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [(1 << 31) - 2, (1 << 32) - 2, (1 << 32) - 1])
def test_ids_past_the_limit(bad):
    tri = (np.array([0, 1, 0], np.uint32), np.array([1, 2, 2], np.uint32), np.ones(3, np.int8))
    big = (tri[0], np.array([1, 2, bad], np.uint32), tri[2])
    with stc.Context(0) as c:
        for persistent in (False, True, True, True):
            with pytest.raises(stc.StcError) as e:
                c.count_batch([tri, big, tri], persistent=persistent)
            assert e.value.status == _capi.STC_ERR_LIMIT
        # A group that is replayed, then the same arrays with a large id.
        src, dst, sign = (np.concatenate([tri[k], tri[k]]) for k in range(3))
        off = np.array([0, 3, 6], np.uint64)
        for _ in range(4):
            got = c.count_batch_packed(src, dst, sign, off)
            assert [x.as_tuple() for x in got] == [oracle.count_arrays(*tri)] * 2
        dst[2] = bad
        with pytest.raises(stc.StcError) as e:
            c.count_batch_packed(src, dst, sign, off)
        assert e.value.status == _capi.STC_ERR_LIMIT
