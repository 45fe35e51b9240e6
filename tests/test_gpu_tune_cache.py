"""Settings that an earlier engine stored, for which alpha and ctas_per_sm meant
something else, are not taken from a cache file."""
import pytest

import turbobfs_gb300 as tb
from turbobfs_gb300 import graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["rmat", "grid"])
def test_lines_of_another_version_are_not_used(gpu_available, tmp_path, kind):
    h = graphs.rmat(12, 16, seed=3) if kind == "rmat" else graphs.grid(40, seed=3)
    roots = graphs.pick_roots(h, 2, seed=3)
    new, old = tmp_path / "new.txt", tmp_path / "old.txt"
    g = tb.Graph.from_host_csc(h)
    g.autotune(roots, cache=str(new))
    key = new.read_text().split()[0]
    old_key = key[:key.index("_sym") + 4]  # the profile alone, as it was
    old.write_text(f"{old_key} 99 18 0.5 1 1\n")
    t = g.autotune(roots, cache=str(old))
    again = g.autotune(roots, cache=str(old))
    g.close()
    assert not t["from_cache"] and t["alpha"] != 99.0
    assert again["from_cache"] and again["alpha"] == t["alpha"]
