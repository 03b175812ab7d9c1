"""The tuner's cache when an entry does not fit the kernels, and its Lanczos candidates."""
import json
import re

import numpy as np
import pytest

from codyfortran_gb300 import init as I
from codyfortran_gb300 import spec as S

pytestmark = pytest.mark.gpu


def _engine(precision):
    from codyfortran_gb300.engine import Engine
    sp = S.helium_fedvr(60, 6, 4)
    sp.xmin, sp.xmax = -60.0, 60.0
    e = Engine(sp, precision, max_krylov=12)
    c = np.ones(e.nC, dtype=complex) / np.sqrt(e.nC)
    e.upload(I.pack_state(c, I.seeded_gaussian_orbitals(sp, e.x, e.w, 3)))
    return e


@pytest.mark.parametrize("entry", [{"W": [80, 0, 1]}, {"Z": [17, 1, 1]}, {"H2": [64, 0, 10**6]}, {"lz_blocks": 10**6}])
def test_an_entry_that_does_not_fit_counts_as_absent(tmp_path, entry):
    """A tile width without a kernel for six slices, splits beyond the buffers: tuned afresh and replaced."""
    cache = tmp_path / "tiles.jsonl"
    e = _engine("mixed_fx6")
    rep = e.autotune(cache)
    line = json.loads(cache.read_text())
    cache.write_text(json.dumps({**line, **entry}) + "\n")
    rep2 = e.autotune(cache)
    again = json.loads(cache.read_text())
    e.close()
    assert rep["source"] == rep2["source"] == "tuned" and rep["key"] == rep2["key"]
    for k, v in entry.items():
        assert again[k] != v


def test_the_key_names_the_slices_and_the_kernels_version():
    keys = {}
    for precision in ("fp64", "mixed", "mixed_fx", "mixed_fx6"):
        e = _engine(precision)
        keys[precision] = e.autotune(None, force=True)["key"]
        e.close()
    assert all(re.search(r";fx=\d+,\d+,v\d+;", k) for k in keys.values())
    assert len({re.search(r"fx=[^;]*", k).group(0) for k in keys.values()}) >= 3


def test_the_lanczos_candidates_run_the_form_that_they_are_for():
    """A launch a pass: at least three per Krylov order, where a context's own steps take one in all."""
    e = _engine("fp64")
    e.launch_count(reset=True)
    rep = e.autotune(None, force=True)
    n = e.launch_count()
    e.close()
    assert n >= 3 * 12 * 2 * len(rep["lz_candidates"])
