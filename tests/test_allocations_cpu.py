"""Every allocation a context makes after its creation gives up the bond terms'
memory, which is not needed, before it fails: none goes to cudaMalloc itself."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "exastamp_gb300", "csrc")


def test_context_allocations_go_through_dev_malloc():
    allowed = {"dev_malloc", "ensure_bpair", "gbmd_create"}
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu") or name in ("gbmd_batch.cu",):  # a batch has no context
            continue
        with open(os.path.join(CSRC, name)) as fh:
            src = re.sub(r"//[^\n]*", "", fh.read())
        inside = None
        for line in src.splitlines():
            m = re.match(r"(?:static |inline )?[\w:]+\*? \*?(\w+)\([^;]*$", line)
            if m:
                inside = m.group(1)
            if "cudaMalloc(" in line:
                assert inside in allowed, (name, inside, line)
