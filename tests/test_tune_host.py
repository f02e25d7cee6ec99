"""The launch tuner's choice and store on the CPU (tune/store.rs, driver/mod.rs, config.rs:8-75),
through `avd_tune_variant_for_test`, which times variant v as the given milliseconds instead of a
launch: Auto keeps the fastest (the baseline keeps ties) and writes one JSON line per key, Cached
reads the store and otherwise answers the baseline, Off always answers the baseline, and a later
process (the remembered results dropped) reads the stored choice without timing again."""

import ctypes as C
import json

import pytest

AUTO, CACHED, OFF = 0, 1, 2


def pick(lib, mode, store, key, times):
    arr = (C.c_float * len(times))(*times)
    return lib.avd_tune_variant_for_test(mode, store.encode() if store else None, key.encode(), len(times), arr)


@pytest.fixture
def store(tmp_path, lib):
    lib.avd_tune_forget()
    yield str(tmp_path)
    lib.avd_tune_forget()


def lines(path):
    with open(path + "/av-denoise-b200-tune.jsonl") as f:
        return [json.loads(line) for line in f if line.strip()]


def test_auto_keeps_the_fastest_and_stores_it(lib, store):
    assert pick(lib, AUTO, store, "site a", [1.0, 0.7, 0.9]) == 1
    rows = lines(store)
    assert len(rows) == 1 and rows[0]["format"] == 1 and rows[0]["variant"] == 1
    assert rows[0]["key"].endswith("site a") and rows[0]["ms"] == pytest.approx([1.0, 0.7, 0.9])
    # Remembered: asked again with other timings, the first answer stands and nothing is appended.
    assert pick(lib, AUTO, store, "site a", [0.1, 5.0, 5.0]) == 1
    assert len(lines(store)) == 1


def test_the_baseline_keeps_ties_and_failed_variants_are_skipped(lib, store):
    assert pick(lib, AUTO, store, "tie", [0.5, 0.5, 0.6]) == 0
    assert pick(lib, AUTO, store, "failed", [-1.0, 0.8, 0.4]) == 2
    assert pick(lib, AUTO, store, "all failed", [-1.0, -1.0]) == 0


def test_cached_reads_the_store_of_an_earlier_process(lib, store):
    assert pick(lib, AUTO, store, "shape", [2.0, 1.0, 3.0]) == 1
    lib.avd_tune_forget()  # a new process: only the file remains
    assert pick(lib, CACHED, store, "shape", [0.1, 9.0, 9.0]) == 1
    assert pick(lib, CACHED, store, "unknown shape", [9.0, 0.1]) == 0
    assert len(lines(store)) == 1


def test_off_and_single_variant_sites_answer_the_baseline(lib, store):
    assert pick(lib, OFF, store, "off", [9.0, 0.1]) == 0
    assert pick(lib, AUTO, store, "one", [9.0]) == 0
    import os

    assert not os.path.exists(store + "/av-denoise-b200-tune.jsonl")


def test_without_a_store_results_last_for_the_process(lib, store):
    assert pick(lib, AUTO, None, "memory", [3.0, 1.0]) == 1
    assert pick(lib, CACHED, None, "memory", [0.1, 9.0]) == 1
    lib.avd_tune_forget()
    assert pick(lib, CACHED, None, "memory", [0.1, 9.0]) == 0


def test_tuning_config_maps_onto_the_abi():
    from conftest import avd

    t = avd.TuningConfig(mode="cached", store="/tmp/x")._c()
    assert t.mode == CACHED and t.store == b"/tmp/x" and t.deterministic == 0
    with pytest.raises(avd.InvalidOptions):
        avd.TuningConfig(mode="sometimes")._c()


IDENTITY_PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include <string>
#include <cuda_runtime.h>
#include "tune.h"

static int current = 0, queries = 0, fail = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
extern "C" cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int dev) {
    ++queries;
    if (fail) return cudaErrorInvalidValue;
    std::snprintf(p->name, sizeof(p->name), "GPU %d", dev);
    p->major = 10;
    p->minor = 0;
    p->multiProcessorCount = 100 + dev;
    return cudaSuccess;
}

int main() {
    fail = 1;
    if (avd::tune_device_identity() != "unknown") return 1;
    fail = 0;
    for (int round = 0; round < 3; ++round)
        for (int dev : {0, 3}) {
            current = dev;
            if (avd::tune_device_identity() != "GPU " + std::to_string(dev) + " sm_100 x" + std::to_string(100 + dev))
                return 2;
        }
    return queries == 3 ? 0 : 3;  // the one that failed, then one per device
}
"""


def test_the_device_is_identified_once(tmp_path):
    """The properties query takes milliseconds, and every engine asks for its store key at its first
    window: one query per device, against a stand-in of the runtime."""
    import subprocess
    from pathlib import Path

    root = Path(__file__).resolve().parent.parent
    csrc = root / "av-denoise_b200" / "csrc"
    src, exe = tmp_path / "identity.cpp", tmp_path / "identity"
    src.write_text(IDENTITY_PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{csrc}", f"-I{root / 'include'}", "-I/usr/local/cuda/include", str(src),
                    str(csrc / "tune.cpp"), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
