"""bench.py prints a captured DRAM traffic beside its E half only when the capture is
of that kernel, named with its template arguments in the kernel's own order."""
import json
import os
import re
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402


def test_committed_capture_is_of_the_benched_kernel():
    with open(os.path.join(ROOT, "profiles", "traffic_e_half.json")) as f:
        t = json.load(f)
    assert t["kernel"] == bench.E_HALF_KERNEL
    assert bench.traffic_of(bench.E_HALF_KERNEL) == t["full_size"]["dram_read"] + t["full_size"]["dram_write"]
    # e_half_kernel<type, cells per thread, mode, poles, ..>, two cells per thread in rows of 256
    src = open(os.path.join(ROOT, "mpulse_b200", "csrc", "mp_step_kernels.cu")).read()
    assert re.search(r"template <typename T, int V, int MODE, int NP, [^>]*>\s*__global__[^;{]*\be_half_kernel", src)
    assert re.fullmatch(r"e_half_kernel<float, 2, PLRC_NONLIN, 2>", bench.E_HALF_KERNEL)


def test_capture_of_another_kernel_is_not_used(tmp_path):
    p = tmp_path / "traffic.json"
    p.write_text(json.dumps({"kernel": "e_half_kernel<float, PLRC_NONLIN, 2>", "bytes_per_launch": 4180000000}))
    assert bench.traffic_of(bench.E_HALF_KERNEL, str(p)) is None
    assert bench.traffic_of(bench.E_HALF_KERNEL, str(tmp_path / "absent.json")) is None
