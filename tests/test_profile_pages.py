"""The figures bench.py takes from profiles/ belong to the kernels that run now."""
import re
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_pages_name_kernels_that_exist():
    source = "\n".join(p.read_text() for p in (ROOT / "myrt_b200" / "csrc").glob("*.cu*"))
    kernels = set(re.findall(r"\b(k_[a-z0-9_]+)", source))
    for page in sorted((ROOT / "profiles").glob("*.md")):
        named = set(re.findall(r"\b(k_[a-z0-9_]*[a-z0-9])\b", page.read_text()))
        assert named <= kernels, (page.name, sorted(named - kernels))


def test_fp32_roofline_only_of_the_kernel_that_was_counted():
    sys.path.insert(0, str(ROOT))
    import bench

    fold, other = bench._sdf_fp32_roofline(compiled=True), bench._sdf_fp32_roofline(compiled=False)
    assert fold["achieved"] == bench.profiled_sdf_fp32_tflops() and 0 < fold["frac"] < 1
    assert other["achieved"] is None and other["frac"] is None
    assert "interpreter" not in fold["source"]
