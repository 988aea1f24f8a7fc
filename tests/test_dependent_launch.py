"""Who decides about programmatic dependent launch: the process's explicit choice, then the thread's scope, then the default (off)."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

from mary_b200 import _native

ROOT = Path(__file__).resolve().parents[1]
CHILD = """
import sys
from mary_b200.ops import cuda as K
state = lambda: K.lib().mary_pdl_state()
if sys.argv[1] != "-":
    K.set_pdl(sys.argv[1] == "1")
out = [state()]
with K.chained:
    out.append(state())
    with K.chained:
        out.append(state())
out.append(state())
K.lib().mary_pdl_scope(0)            # a choice of the thread's own outlasts a scope
with K.chained:
    out.append(state())
out.append(K.lib().mary_pdl_scope(-1))
print(*out)
"""


@pytest.mark.skipif(not _native.kernels_available(), reason="kernel library not built")
@pytest.mark.parametrize("env,call,outside,inside", [(None, "-", 0, 1), ("0", "-", 0, 0), ("1", "-", 1, 1), (None, "0", 0, 0), (None, "1", 1, 1), ("1", "0", 0, 0),
                                                     ("0", "1", 1, 1)])
def test_an_explicit_choice_holds_inside_the_scope(env, call, outside, inside):
    e = {k: v for k, v in os.environ.items() if k != "MARY_PDL"}
    e["PYTHONPATH"] = str(ROOT)
    if env is not None:
        e["MARY_PDL"] = env
    r = subprocess.run([sys.executable, "-c", CHILD, call], env=e, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stdout.split() == [str(v) for v in (outside, inside, inside, outside, inside, 0)]
