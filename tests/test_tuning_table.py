"""A caller's tuning table decides about bucket lists, also for a lone range of
one wave of segments; the library's own table, set back, is its own again."""
import json
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

# The lists of [10^12, 10^12 + 10^8) from 221184 on take 18 MB (152 segments of
# 22016 bytes, expected entries 8 * 22016 * sum(1/p) = 20 000 each, 4 bytes, with
# their margin), which the engine allocates when a call first uses them.
PROBE = r"""
import ctypes
import json
import torch
import voss_gb300 as vg
from voss_gb300 import _capi
from voss_gb300.autotune import TuneEntry, U64_MAX, set_table
lib = _capi._lib
a, b = 10**12, 10**12 + 10**8
n = ctypes.c_uint32()
own = (TuneEntry * 64)()
assert lib.voss_gb300_get_tuning(64, own, ctypes.byref(n)) == 0
own = [tuple(getattr(e, f) for f, _ in TuneEntry._fields_) for e in own[:n.value]]

def used(table):
    set_table(lib, table)
    before = torch.cuda.mem_get_info()[0]
    st = vg.range_stats(a, b)
    return (before - torch.cuda.mem_get_info()[0]) >> 20, (st.count, st.max_gap, st.max_gap_start, st.pi_4_1)

set_table(lib, own)
plain = vg.range_stats(a, b)                   # the engine's buffers for runs without lists
print(json.dumps([used(own), used([(U64_MAX, U64_MAX, 222848, 2048, 0)]), used([(U64_MAX, U64_MAX, 222848, 2048, 221184)])]))
"""


def test_a_callers_split_takes_lists(vg):
    out = subprocess.run([sys.executable, "-c", PROBE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    (own_mb, own), (none_mb, none), (lists_mb, lists) = json.loads(out.stdout)
    assert own == none == lists
    assert own_mb < 8 and none_mb < 8 and lists_mb >= 16, out.stdout
