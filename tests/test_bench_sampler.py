"""The clock record of a timed region that is shorter than NVML's first answers, with an NVML of the test's own."""

import sys
import time
import types

import bench


def test_a_short_region_is_sampled_from_its_beginning(monkeypatch):
    asked = {}

    def answer(name, value):
        def query(*_):
            asked[name] = asked.get(name, 0) + 1
            if asked[name] == 1:
                time.sleep(0.05)
            return value

        return query

    nvml = types.ModuleType("pynvml")
    nvml.NVML_CLOCK_SM = 1
    nvml.nvmlInit = lambda: time.sleep(0.02)
    nvml.nvmlDeviceGetHandleByIndex = lambda index: index
    nvml.nvmlDeviceGetMaxClockInfo = lambda handle, kind: 1965
    nvml.nvmlDeviceGetClockInfo = answer("clock", 1900)
    nvml.nvmlDeviceGetCurrentClocksEventReasons = answer("reasons", 0x4)
    monkeypatch.setitem(sys.modules, "pynvml", nvml)
    sampler = bench.ClockSampler(0)
    sampler.begin()
    time.sleep(0.04)
    sampler.stop_flag.set()
    sampler.join(timeout=2)
    summary = sampler.summary()
    assert summary["samples"] >= 3  # of about twenty: a loaded host may wake a thread late
    assert summary["sm_mhz"] == 1900 and summary["sm_max_mhz"] == 1965 and summary["reasons"] == ["sw_power_cap"]


def test_an_nvml_that_fails_does_not_hold_the_region_up(monkeypatch):
    nvml = types.ModuleType("pynvml")
    nvml.NVML_CLOCK_SM = 1
    nvml.nvmlInit = lambda: None
    nvml.nvmlDeviceGetHandleByIndex = lambda index: index
    nvml.nvmlDeviceGetMaxClockInfo = lambda handle, kind: 1965

    def fails(*_):
        raise RuntimeError("no clocks")

    nvml.nvmlDeviceGetClockInfo = fails
    monkeypatch.setitem(sys.modules, "pynvml", nvml)
    sampler = bench.ClockSampler(0)
    start = time.perf_counter()
    sampler.begin()
    assert time.perf_counter() - start < 5
    sampler.stop_flag.set()
    sampler.join(timeout=2)
    assert "no clocks" in sampler.summary()["error"]
