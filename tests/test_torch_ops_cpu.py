"""CPU tests of the native half of capi.py: what happens to the arguments before anything is launched."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_FRESH = """
import torch
from amdmigraphx_b200 import capi

events = []

class Item:
    def __init__(self, name, value):
        self.name, self.value = name, value
    def __index__(self):
        events.append(("read", self.name))
        return self.value
    def __float__(self):
        events.append(("read", self.name))
        return float(self.value)
    def __del__(self):
        events.append(("freed", self.name))

class Fresh:
    '''A sequence that keeps none of its items.'''
    def __init__(self, name, values):
        self.name, self.values = name, values
    def __len__(self):
        return len(self.values)
    def __getitem__(self, i):
        v = self.values[i]
        return Item(f"{self.name}{i}", v) if isinstance(v, int) else v

add = Fresh("insn", ("add", capi.F16, Fresh("src", (0, 1)), 0))
try:
    # the second input does not have the result's shape: refused after everything of the first was read
    capi.pointwise([torch.zeros(2, 3, dtype=torch.float16), torch.zeros(7, dtype=torch.float16)], [add], Fresh("len", (2, 3)))
    raise SystemExit("accepted")
except AssertionError:
    pass
try:
    # an unknown result type is refused after all instructions were read
    capi.pointwise([torch.zeros(2, 3, dtype=torch.float16)] * 2, [Fresh("insn", ("add", 77, Fresh("src", (0, 1)), 0))],
                   Fresh("len", (2, 3)))
    raise SystemExit("accepted")
except KeyError:
    pass
names = [n for _, n in events]
want = {"len0", "len1", "insn1", "insn3", "src0", "src1"}
assert want <= set(names), names
for n in want:
    own = [e for e, m in events if m == n]
    assert own == ["read", "freed"] * (len(own) // 2), (n, own)
print("ok")
"""


def test_pointwise_holds_items_that_a_sequence_makes_on_the_fly():
    """Lengths, instructions and operands may come from any sequence, arrays and ranges included, whose items
    exist only while somebody holds them: each is read before it is released.  (In a process of its own: reading a
    released one may end it.)"""
    r = subprocess.run([sys.executable, "-c", _FRESH], capture_output=True, text=True, cwd=ROOT, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout, r.stderr[-2000:])
