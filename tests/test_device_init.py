"""Device memory that the host fills (status records, pointer tables, new blocks) is filled before a kernel can read it."""
import pathlib
import re
import subprocess
import sys

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "symm_mem_recipes_b200" / "csrc"


def test_the_host_waits_for_what_it_writes_on_the_legacy_stream():
    """cudaMemset, and cudaMemcpy from pageable memory, may return before the device has the bytes, and kernels on
    non-blocking streams are not ordered after them: a wait follows each (or the next line's write, then a wait)."""
    bad, seen = [], 0
    for path in sorted(p for ext in ("*.cu", "*.cpp") for p in CSRC.rglob(ext)):
        lines = [ln for ln in path.read_text().splitlines() if not ln.strip().startswith("//")]
        writes = [i for i, ln in enumerate(lines) if re.search(r"cudaMemset\(\w|cudaMemcpy\(.*HostToDevice", ln)]
        for i in writes:
            seen += 1
            after = i + 1
            while after in writes:
                after += 1
            if "Synchronize(" not in lines[after]:
                bad.append(f"{path.name}: {lines[i].strip()}")
    assert seen >= 3 and not bad, bad


_FIRST_CALL_IN_A_CAPTURE = """
import torch
import symm_mem_recipes_b200 as smr
from symm_mem_recipes_b200.parallel import symm_mem
a = torch.randn(300, 512, device="cuda", dtype=torch.bfloat16)
b = torch.randn(384, 512, device="cuda", dtype=torch.bfloat16)
want = a.float() @ b.float().t()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    c = smr.matmul(a, b)
g.replay()
symm_mem.check_status("cuda")
assert bool(((c.float() - want).abs() <= want.abs() * 2.0 ** -6 + 2e-1).all())
print("first call ok")
"""


@pytest.mark.gpu
def test_first_call_of_a_process_may_be_captured():
    out = subprocess.run([sys.executable, "-c", _FIRST_CALL_IN_A_CAPTURE], cwd=CSRC.parent.parent, capture_output=True,
                         text=True, timeout=200)
    assert out.returncode == 0 and "first call ok" in out.stdout, out.stderr[-2000:]


def test_launchers_ask_the_device_for_its_sms():
    """148, or a multiple of it, in a launcher would size the grids of one chip."""
    bad = []
    for path in sorted((CSRC / "kernels").rglob("*.cu")):
        for n, ln in enumerate(path.read_text().splitlines(), 1):
            if re.search(r"\b(148|296|592|9472)\b", ln.split("//")[0]):
                bad.append(f"{path.name}:{n}: {ln.strip()}")
    assert not bad, bad
