"""The transforms' exchange buffers are addressed by XORs on bits 2-6 of
shared-memory addresses (csrc/ntt_joint.cuh), so every buffer must start on 128
bytes: the declarations that decide it, in every source that uses them."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "inspire-rs_gb300", "csrc")


def test_exchange_buffers_are_declared_aligned():
    used = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            text = f.read()
        names = set(re.findall(r"\bjx_addr\((\w+)", text))
        if not names:
            continue
        used += 1
        for line in re.findall(r"extern __shared__[^;]*;", text):
            assert "__align__(128)" in line, (os.path.basename(path), line)
        for line in re.findall(r"(?<!extern )__shared__[^;]*;", text):
            name = re.search(r"(\w+)(\[[^\]]*\])*;$", line).group(1)
            if name in names:
                assert "__align__(128)" in line, (os.path.basename(path), line)
    assert used >= 6
