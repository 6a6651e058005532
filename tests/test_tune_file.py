"""A handle whose tuning choices come from a file (BDC_TUNE_FILE) runs the
same kernels as the handle that measured and wrote them."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n,k", [(14, 12), (20, 10), (26, 14)])
def test_pinned_handle_repeats_the_measured_one(bdc, tmp_path, monkeypatch, n, k):
    """The second handle takes no measurement during set-up.  The same kernels
    add in the same order, so the iterates agree to the last bit."""
    monkeypatch.setenv("BDC_TUNE_FILE", str(tmp_path / "tune.txt"))
    got = []
    for _ in range(2):
        with bdc.Engine(n, k, engine="factored") as E:
            E.set_uniform()
            st = E.iterate(2)
            got.append((E.get_p(), st["upper_bound"], st["rate"], (tmp_path / "tune.txt").read_text()))
    np.testing.assert_array_equal(got[0][0], got[1][0])
    assert got[0][1:] == got[1][1:]
