"""The benchmark's arithmetic on kernel times: no GPU needed."""

import inspect
import sys
import time
import types

import bench


def test_rounds_of_a_call_add_up():
    # 20 steps of one compression and two rounds of expansion and attention, of which 30 attention launches were recorded
    ms = bench.kernel_ms_per_step([2.0, 0.0, 8.0, 45.0, 0.0], [20, 0, 40, 30, 0], [1, 0, 2, 2, 0])
    assert ms == [0.1, 0.0, 0.4, 3.0, 0.0]


def test_decode_section_names_its_kernels():
    source = inspect.getsource(bench.decode_section)
    assert '"prepare_queries"' in source and "expand" not in source


def test_clocks_are_sampled_in_short_regions(monkeypatch):
    # a stand-in for NVML that takes longer to open than the region lasts
    nvml = types.ModuleType("pynvml")
    nvml.nvmlInit = lambda: time.sleep(0.3)
    nvml.nvmlDeviceGetHandleByIndex = lambda i: i
    nvml.NVML_CLOCK_SM = 1
    nvml.nvmlDeviceGetMaxClockInfo = nvml.nvmlDeviceGetClockInfo = lambda h, kind: 1965
    nvml.nvmlDeviceGetCurrentClocksThrottleReasons = lambda h: 0
    for i, name in enumerate(("HwSlowdown", "HwThermalSlowdown", "SwThermalSlowdown", "SwPowerCap", "HwPowerBrakeSlowdown")):
        setattr(nvml, "nvmlClocksThrottleReason" + name, 1 << i)
    monkeypatch.setitem(sys.modules, "pynvml", nvml)
    sampler = bench.ClockSampler(0)
    sampler.start()
    time.sleep(0.05)
    assert sampler.finish()["sm_mhz"] == 1965
