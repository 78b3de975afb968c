"""The allocation-free cell sort at the edges of its tiles (1024 and 2048 keys,
with the change between them), of the offsets' blocks (256 elements) and on keys
that are all alike, against numpy's stable argsort: exact."""
import numpy as np
import pytest
import torch

from test_zz_no_alloc import _call, _entry, _expected

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ne", [1, 255, 256, 257, 70000])
def test_sort_edges(ne):
    fn = _entry()
    rng = np.random.default_rng(ne)
    line = torch.cuda.get_device_properties(0).multi_processor_count * 1024
    for n in (0, 1, 31, 1023, 1024, 1025, 2049, line, line + 1):
        for keys in (rng.integers(-1, ne + 2, n), np.full(n, ne - 1), np.full(n, -1), np.sort(rng.integers(0, ne, n))):
            got = _call(torch, fn, np.asarray(keys, dtype=np.int32), ne)
            for g, w, name in zip(got, _expected(np.asarray(keys, dtype=np.int64), ne), ("keys", "perm", "start")):
                np.testing.assert_array_equal(g, w, err_msg="%s n %d" % (name, n))
