"""Which path a prediction of a few rows takes: one launch as long as reading the support vectors once per eight rows costs
less than the general path's launches (1.6e7 entries), whatever the caller's row_ptr has told the handle so far."""
import fake_device
import pytest

from test_full_device_cpu import PREDICT, runtime  # noqa: F401


@pytest.mark.parametrize("loc", ["DEVICE", "HOST"])
@pytest.mark.parametrize("per_row,rows,one_launch", [(500, 16, False), (500, 8, True), (70, 16, True), (399, 16, True),
                                                     (401, 16, False)])
def test_few_rows_of_sparse_data(runtime, loc, per_row, rows, one_launch):  # noqa: F811
    fake_device.run_python(runtime, PREDICT + """
s, h, keep = csr(20000, 5000, %d, loc=%s)
check(s)
s, h2, batch = csr(%d, 5000, 70)
F.fake_reset_counts()
check(predict(h, 20000, %d, csr=batch))
assert (F.fake_launches() == 1) == %s, F.fake_launches()
""" % (per_row, loc, rows, rows, one_launch))
