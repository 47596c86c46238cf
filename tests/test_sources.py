"""Rules of the CUDA sources that the compiler does not check."""
import glob
import os
import re

from conftest import ROOT


def test_warp_wide_asm_is_volatile():
    """An inline asm without `volatile` may be moved or deleted, into a branch
    that some of a warp's lanes do not take: an instruction that the whole warp
    takes part in (.sync) or that copies memory (cp.async) has to stay where it
    is written."""
    seen = 0
    for path in sorted(glob.glob(os.path.join(ROOT, "pump_gb300", "csrc", "*.cu*"))):
        with open(path) as f:
            src = f.read()
        for m in re.finditer(r"\basm\b(\s+volatile\b)?\s*\(\s*\"([^\"]*)\"", src):
            if ".sync" in m.group(2) or "cp.async" in m.group(2):
                seen += 1
                assert m.group(1), (os.path.basename(path), m.group(2))
    assert seen >= 4
