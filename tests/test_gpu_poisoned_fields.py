"""The tests that stress the kept part of the REV arrays, the lines that the field
can reach and the cleared part of the gradient, once more with the arenas filled
with NaN before each chunk (EE_DEBUG_POISON=1): a sample read without having been
written or cleared turns a dose or gradient into NaN."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_fields_and_chunks_with_poisoned_rev_arenas():
    env = dict(os.environ, EE_DEBUG_POISON="1")
    tests = [f"tests/test_gpu_{t}.py" for t in
             ("field_span", "chunks", "gather_split", "sparse_gradient", "table_span", "plan_chunks")]
    r = subprocess.run([sys.executable, "-m", "pytest", *tests, "-x", "-q", "-m", "gpu", "-p", "no:cacheprovider",
                        "--basetemp", os.path.join(ROOT, ".pytest_tmp", "poison_fields")],
                       cwd=ROOT, env=env, capture_output=True, text=True, timeout=1200)
    print(r.stdout[-3000:])
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-2000:]
