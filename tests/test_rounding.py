"""The kernels round as IEEE does: no approximate instruction forms in the device sources, and no flag asks for them."""
import re
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_no_approximate_arithmetic():
    from sol_b200 import build
    for p in (ROOT / "sol_b200" / "csrc").rglob("*"):
        if p.suffix in (".cu", ".cuh", ".h") and p.name != "probe.cu":   # probe.cu: bandwidth probes only
            found = re.search(r"\.approx\b|__fdividef|__frcp_r[duz]|__(?:exp|log|pow|sin|cos)f\b|\.ftz", p.read_text())
            assert not found, (p.name, found and found.group())
    flags = " ".join(build.NVCC_DEVICE)
    assert "-prec-div=true" in flags and "-prec-sqrt=true" in flags and "-fmad=false" in flags and "fast" not in flags
