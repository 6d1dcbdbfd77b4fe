"""Every device and pinned-host allocation of the library goes through the
counting wrappers of csrc/plan.cpp (lib_malloc and its kind), which the
out-of-memory tests and the live-allocation count rest on."""
import os
import re

from _pkg import PKG_DIR

CSRC = os.path.join(PKG_DIR, "csrc")
RAW = re.compile(r"\bcuda(?:Malloc\w*|HostAlloc|Free\w*)\s*\(")


def _functions(text):
    """(name, body) of the top-level functions whose bodies close in column 0."""
    for m in re.finditer(r"^(?:template <[^>]*> )?static [^\n;(]*?(\w+)\([^;{]*\) \{$(.*?)^\}$", text, re.M | re.S):
        yield m.group(1), m.group(2)


def test_raw_allocation_calls_sit_in_the_wrappers():
    calls = wrapped = 0
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cpp", ".cu", ".cuh", ".h")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        calls += len(RAW.findall(text))
        if f == "plan.cpp":
            wrapped = sum(len(RAW.findall(body)) for name, body in _functions(text) if name.startswith("lib_"))
    assert wrapped >= 4
    assert calls == wrapped, (calls, wrapped)
