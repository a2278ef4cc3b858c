"""The pivot-list check behind bbtc_graph_validate, on the CPU: lists built on
the host pass, and each planted fault is named."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from bbtc_b200 import graphs

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAULTS = {
    "entries_first": "wrong entries",
    "entries_end": "wrong entries",
    "vertex": "wrong entries",
    "pair": "differs from its row",
    "pairs": "differs from its row",
    "word": "differs from its row",
    "span": "differs from its row",
    "bits": "keeps the wrong ids",
    "record_first": "record",
    "record_end": "record outside the row's pairs",
    "index": "entry index names the wrong pivot",
    "missing": "a pivot is missing",
    "surplus": "too many pivots",
    "end_mark": "no end mark",
}


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("pc")
    exe = d / "harness"
    cxx = shutil.which("g++") or shutil.which("c++")
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-I", os.path.join(ROOT, "bbtc_b200", "csrc"),
                    os.path.join(ROOT, "tests", "pivot_check_harness.cpp"), "-o", str(exe)], check=True)

    def run(g, cuts, fault):
        path = d / "g.bin"
        with open(path, "wb") as f:
            np.array([g.n, len(cuts) - 1], np.uint32).tofile(f)
            np.array([g.m], np.uint64).tofile(f)
            for a in (g.indptr, g.indices, cuts):
                np.asarray(a, np.uint32).tofile(f)
        r = subprocess.run([str(exe), str(path), fault], capture_output=True, text=True, timeout=60)
        assert r.returncode == 0, (fault, r.stdout, r.stderr)
        return r.stdout.strip()

    return run


def unoriented(n, max_deg, seed):
    rng = np.random.default_rng(seed)
    rows = [np.unique(rng.integers(0, n, size=int(d))) for d in rng.integers(0, max_deg + 1, size=n)]
    indptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint32)
    return graphs.OrientedCSR(n, indptr, np.concatenate(rows).astype(np.uint32))


GRAPHS = {"oriented": lambda: graphs.rmat(9, 8, seed=3), "unoriented": lambda: unoriented(300, 40, 5)}


@pytest.mark.parametrize("graph", sorted(GRAPHS))
@pytest.mark.parametrize("cuts", ["one", "some", "empty"])
def test_right_lists_pass(harness, graph, cuts):
    g = GRAPHS[graph]()
    c = {"one": [0, g.n], "some": [0, 100, 131, 256, g.n], "empty": [0, 0, 37, 37, g.n + 5]}[cuts]
    assert harness(g, c, "none") == "OK"


@pytest.mark.parametrize("fault", sorted(FAULTS))
@pytest.mark.parametrize("graph", sorted(GRAPHS))
def test_planted_faults_are_named(harness, graph, fault):
    g = GRAPHS[graph]()
    out = harness(g, [0, 100, 131, 256, g.n], fault)
    assert out != "OK" and FAULTS[fault] in out, (fault, out)
