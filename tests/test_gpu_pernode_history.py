"""A solve's bits do not depend on what ran before it in the process: the CTAs of
a per-node kernel, and so the grouping of its sums, are that kernel's own."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import sys, zlib
sys.path.insert(0, {pkg!r})
import torch, sipg_gb300 as sipg

def solve(p, shape):
    op = sipg.Operator(128, p, float(p * p))
    op.set_pernode(shape)
    b = op.rhs("sinsin")
    x = torch.zeros_like(b)
    op.cg(x, b, 1e-30, relative=True, max_it=3)
    return "%08x" % zlib.crc32(x.cpu().numpy().tobytes())

order = [(p, s) for p in (2, 4, 8) for s in {shapes!r}]
print(" ".join("%d:%d:%s" % (p, s, solve(p, s)) for p, s in order))
"""


def test_solves_do_not_depend_on_earlier_launches(sipg):
    import os

    pkg = os.path.dirname(os.path.abspath(sipg.__file__))
    seen = []
    for shapes in ((0, 1), (1, 0)):
        out = subprocess.run([sys.executable, "-c", SCRIPT.format(pkg=pkg, shapes=shapes)], capture_output=True,
                             text=True, timeout=120)
        assert out.returncode == 0, out.stderr[-2000:]
        seen.append(sorted(out.stdout.split()))
    assert seen[0] == seen[1]
