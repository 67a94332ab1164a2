"""The streamed transmit on every grid that has one.  Which plan a grid's transmit keeps
is chosen by timing (at 64^2 to 256^2 mostly the 16-point plan, which does not stream), so
the comparisons of test_gpu_streamed.py run here with the 32-point plan fixed, in a
process of their own: its large calls are above the streaming rule then."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_streamed_with_the_plan_fixed():
    r = subprocess.run([sys.executable, "-m", "pytest", os.path.join(HERE, "test_gpu_streamed.py"), "-q", "-x",
                        "-m", "gpu", "-p", "no:cacheprovider"], env=dict(os.environ, MSK_ROW_PLAN="0"),
                       cwd=os.path.dirname(HERE), timeout=600, capture_output=True, text=True)
    assert r.returncode == 0 and " passed" in r.stdout and "skipped" not in r.stdout, r.stdout[-3000:]
