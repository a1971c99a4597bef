"""A CSR that is refused costs no host memory beyond its arrays: one list of 64
million entries over two vertices (so not strictly sorted below 2) used to size
the degree tables, four times 8 bytes an entry, before it was looked at."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import resource
import numpy as np
import cuts_b200 as cb
q = cb.Query.from_arcs(*cb.named_query_arcs("triangle"))
h = cb.HostGraph.erdos_renyi(100, 0.1, 1)
g = h.upload(0)
g.count(q)
m = 64 << 20
off, adj = np.array([0, m, m], np.uint64), np.ones(m, np.uint32)
before = resource.getrusage(resource.RUSAGE_SELF).ru_maxrss
for args in ((off, adj), (off, adj, off, adj)):
    try:
        cb.Graph.from_csr(2, *args)
        raise SystemExit("accepted")
    except cb.CutsError as e:
        assert e.code == cb.ERR_ARG, e
print((resource.getrusage(resource.RUSAGE_SELF).ru_maxrss - before) >> 10)
"""


def test_refused_list_longer_than_the_graph():
    out = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-800:]
    assert int(out.stdout.split()[-1]) < 512, out.stdout  # MB; the tables took 2,048
