"""The index and search tools against the oracle.

test_formats_gpu.py holds them to the compiled reference; where that is not
there, the oracle's search of the same index file (pinned to the reference,
test_oracle_pin.py) decides.
"""
import os
import re
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from oracle import kgoracle as ko
from test_formats_gpu import _lshkit, _read_lshkit_u32


@pytest.mark.gpu
def test_index_and_search_tools_match_the_oracle(tmp_path):
    binp = os.path.join(ROOT, "kgraph_b200", "bin")
    rng = np.random.default_rng(17)
    X = rng.random((6000, 24), dtype=np.float32)
    Q = rng.random((200, 24), dtype=np.float32)
    _lshkit(tmp_path / "data", X)
    _lshkit(tmp_path / "query", Q)

    def tool(name, *args):
        r = subprocess.run([os.path.join(binp, name)] + [str(a) for a in args], capture_output=True, text=True,
                           timeout=300)
        assert r.returncode == 0, r.stderr
        return r.stdout

    data, idx, query = tmp_path / "data", tmp_path / "g.idx", tmp_path / "query"
    tool("index", data, idx, "-K", 10, "-L", 30, "-S", 8, "--reverse", -1)
    tool("search", data, idx, query, tmp_path / "gs", "-K", 10, "--linear")
    o = ko.Oracle(X, "l2sqr")
    exact = o.bruteforce(Q, 10)[0]
    assert (_read_lshkit_u32(tmp_path / "gs") == exact).all()
    out = tool("search", data, idx, query, tmp_path / "res", "-K", 10, "-P", 30, "--eval", tmp_path / "gs")
    ids, _, _, cost = o.search(ko.read_index(str(idx)), Q, K=10, P=30)
    assert (_read_lshkit_u32(tmp_path / "res") == ids).all()
    m = re.search(r"Time: (\S+) Recall: (\S+) Cost: (\S+)", out)
    assert m and float(m.group(2)) > 0.9 and abs(float(m.group(3)) - float(cost.mean())) < 1e-5


def test_missing_reference_skips():
    """A test that asks for the compiled reference where it is not built is skipped, not failed."""
    with pytest.raises(ko.ReferenceMissing):
        ko.RefLib("no-such-isa")
