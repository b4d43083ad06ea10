"""What the kernels' sources promise the compiler and what their launchers ask of each device, where a run on one GPU that comes out
right shows nothing (no GPU needed)."""
import os
import re
import subprocess

import pytest

from geneinfer_b200.ops.build import CSRC, _nvcc


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def test_the_router_has_one_pointer_to_the_ids_that_it_writes_and_reads():
    """With few tokens the kernel that writes the experts' ids also buckets them: the struct that the bucketing reads them through
    must be the only way to them, and not one that excludes others (``__restrict__``)."""
    text = _source("grouped_product.cu")
    signature = re.search(r"\nroute_kernel\((.*?)\) \{", text, re.S).group(1)
    held = re.search(r"struct RouteAlign \{(.*?)\};", text, re.S).group(1)
    named = set(re.findall(r"\*\s*(\w+)", held))
    assert "ids" in named and "__restrict__" not in held
    written = set(re.findall(r"(?<!const )(?:int|float)\*\s*(?:__restrict__)?\s*(\w+)", signature))
    assert not written & named, "a second way to memory that the bucketing reads or writes"


# The runtime's two calls, faked: the current device is the thread's, device 3 refuses, and every setting is counted by device.
_FAKE_RUNTIME = r"""
#include "device_limit.h"
#include <cstdio>
#include <thread>
#include <vector>
static thread_local int device = 0;
static std::atomic<int> set_on[80], bytes_on[80], errors_read{0};
extern "C" cudaError_t CUDARTAPI cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t CUDARTAPI cudaGetLastError() { ++errors_read; return cudaSuccess; }
extern "C" cudaError_t CUDARTAPI cudaFuncSetAttribute(const void*, cudaFuncAttribute, int bytes) {
    if (device == 3) return cudaErrorInvalidValue;
    ++set_on[device];
    bytes_on[device] = bytes;
    return cudaSuccess;
}
#define CHECK(x) if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; }
int main() {
    static gi::SharedLimit first, second;
    for (int round = 0; round < 3; ++round)
        for (int d : {0, 1, 63, 70}) {
            device = d;
            CHECK(first.allow(nullptr, 100000 + d) == cudaSuccess && bytes_on[d] == 100000 + d);
        }
    CHECK(set_on[0] == 1 && set_on[1] == 1 && set_on[63] == 1 && set_on[70] == 3 && errors_read == 0);
    device = 1;                                            // another kernel's limit is its own
    CHECK(second.allow(nullptr, 7) == cudaSuccess && set_on[1] == 2 && bytes_on[1] == 7);
    device = 3;                                            // a refusal is reported each time, and not left for the next launch
    CHECK(first.allow(nullptr, 1) == cudaErrorInvalidValue && first.allow(nullptr, 1) == cudaErrorInvalidValue && errors_read == 2);
    std::vector<std::thread> threads;
    static gi::SharedLimit shared;
    std::atomic<int> wrong{0};
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&, t] {
            device = 10 + t % 4;
            for (int i = 0; i < 1000; ++i)
                if (shared.allow(nullptr, 5) != cudaSuccess || set_on[device] < 1) ++wrong;
        });
    for (auto& t : threads) t.join();
    CHECK(wrong == 0);
    return 0;
}
"""


def test_a_kernels_shared_memory_limit_is_set_on_every_device(tmp_path):
    source = tmp_path / "limits.cpp"
    source.write_text(_FAKE_RUNTIME)
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))), "include")
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", CSRC, "-I", include, str(source), "-o", str(tmp_path / "limits")], check=True)
    done = subprocess.run([str(tmp_path / "limits")], stdout=subprocess.PIPE, text=True)
    assert done.returncode == 0, done.stdout


@pytest.mark.parametrize("name", ["gemm_f32.cu", "grouped_product.cu", "linear_recurrence.cu"])
def test_no_launcher_remembers_for_the_process_what_belongs_to_a_device(name):
    """What the 32-bit path launches: it runs on whichever device is current, of several in a process."""
    assert not re.search(r"static (?:const )?(?:bool|cudaError_t) \w+\s*=", _source(name))
