"""Host-side pieces of bench.py that decide what a bench line reports, on CPU:
the clock summary (median SM clock, max clock, throttle reasons seen during
the timed region) from NVML samples and from nvidia-smi lines."""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402


def test_clock_summary_from_nvml_samples():
    c = bench.ClockSampler(0)
    B = bench.ClockSampler.BITS
    c.samples = [(1965.0, 1965.0, 0), (1800.0, 1965.0, B["sw_power_cap"]), (1900.0, 1965.0, 0x1),
                 (1950.0, 1965.0, B["hw_slowdown"] | B["sw_power_cap"])]
    s = c.summary()
    assert s["sm_mhz"] == pytest.approx(1925.0)
    assert s["sm_max_mhz"] == 1965.0
    # bit 0x1 (GPU idle) is not a throttle reason the bench reports
    assert s["reasons"] == ["hw_slowdown", "sw_power_cap"]
    assert s["samples"] == 4 and s["source"] == "nvml"


def test_clock_summary_from_nvidia_smi_lines():
    c = bench.ClockSampler(0)
    c.lines = [
        "0, 1965, 1965, 612.30, 0x0000000000000000, Not Active, Not Active, Not Active, Not Active",
        "0, 1312, 1965, 999.80, 0x0000000000000004, Not Active, Not Active, Not Active, Active",
        "0, 1500, 1965, 800.00, 0x0000000000000020, Not Active, Not Active, Active, Not Active",
        "0, [N/A], 1965, 800.00, 0x0, Not Active, Not Active, Not Active, Not Active",
        "garbage line",
    ]
    s = c.summary()
    assert s["sm_mhz"] == 1500.0
    assert s["sm_max_mhz"] == 1965.0
    assert s["reasons"] == ["sw_power_cap", "sw_thermal_slowdown"]
    assert s["samples"] == 3 and s["source"] == "nvidia-smi"


def test_clock_summary_without_samples():
    s = bench.ClockSampler(0).summary()
    assert s["sm_mhz"] is None and s["sm_max_mhz"] is None and s["reasons"] == [] and s["samples"] == 0


def test_counted_kernels_exist():
    """The lines that report own launches as a fixed number a step name the kernels they count: all of them are kernels
    of the library, and as many as the factor says (a number before a name repeats it)."""
    import glob
    import re

    src = "".join(open(f).read() for f in glob.glob(os.path.join(ROOT, "pbbsbench_b200", "csrc", "*.cu")))
    kernels = set(re.findall(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s+)?(\w+)\s*\(", src))
    text = open(os.path.join(ROOT, "bench.py")).read()
    counted = re.findall(r"((?:^ *#[^\n]*\n)+) *\"gpu_launches\": (\d+) \* args\.steps", text, flags=re.M)
    assert len(counted) >= 3
    for comment, factor in counted:
        named = re.findall(r"(?:(\d+) )?\b((?:k|jump|check|strip)_\w+)", comment)
        assert named and {k for _, k in named} <= kernels, comment
        assert sum(int(c or 1) for c, _ in named) == int(factor), comment
