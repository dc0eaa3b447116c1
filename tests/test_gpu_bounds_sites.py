"""The bounds-checked build on the calls of tests/bounds_workload_sites.py: no checked access leaves its buffer, every
site of the library makes a test (among them the differentiation form's, the float images' taps, the stored sum and the
caller's own maps), and the outputs are the product library's: bit for bit, or for sums of atomics, which have no fixed
order, to 1e-4 of their norm (some thousand FP32 terms a pixel, whose roundings of 2^-24 add up like their root; the
loss and the poses sum in double precision)."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def run(lib, path):
    env = dict(os.environ, PM_STEREO_LIB=lib)
    r = subprocess.run([sys.executable, os.path.join(ROOT, "tests", "bounds_workload_sites.py"), str(path)],
                       env=env, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout + r.stderr
    return np.load(path)


def test_every_site_is_reached_and_stays_in_bounds(pm_lib, tmp_path):
    from probabilistic_mapping_b200 import _lib, build
    checked = run(build.LIB_CHECKED, tmp_path / "checked.npz")
    product = run(build.LIB, tmp_path / "product.npz")
    assert (checked["bounds_status"] == _lib.PM_OK).all()
    assert (product["bounds_status"] == _lib.PM_ERR_UNSUPPORTED).all()
    assert int(checked["bounds"][0]) == 0, f"out-of-range accesses: site, index, extent = {checked['bounds'][1:]}"
    reached, sites = (int(x) for x in checked["bounds_sites"])
    assert sites and reached == sites, f"sites without a test: {[s for s in range(64) if (sites & ~reached) >> s & 1]}"
    keys = [k for k in product.files if not k.startswith("bounds")]
    assert len(keys) > 40 and set(keys) == set(k for k in checked.files if not k.startswith("bounds"))
    for k in keys:
        a, b = product[k], checked[k]
        assert a.shape == b.shape, k
        if k.startswith("~"):
            assert np.linalg.norm(a) > 0 and np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(a), k
        else:
            assert (a.view(np.uint8) == b.view(np.uint8)).all(), k
