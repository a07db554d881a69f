"""What the CUDA sources' host side promises, checked without a GPU."""
import glob
import os
import re
import shutil
import subprocess

import pytest

from tiny_llm_b200.ops import build


def sources():
    return {os.path.basename(f): open(f).read()
            for f in sorted(glob.glob(os.path.join(build.CSRC, "*.cu")) + glob.glob(os.path.join(build.CSRC, "*.cuh")))}


PER_DEVICE = r"""
#include <thread>
#include <vector>
#include "per_device.h"
#define CHECK(x) do { if (!(x)) return __LINE__; } while (0)
int main() {
  static tllm::PerDeviceLimit limit;
  int calls = 0;
  auto fine = [&] { ++calls; return 0; };
  for (int dev = 0; dev < 4; ++dev) {               // every ordinal is set up, once
    for (int i = 0; i < 3; ++i) CHECK(limit.raise(dev, 100, fine) == 0);
    CHECK(calls == dev + 1);
  }
  calls = 0;
  CHECK(limit.raise(2, 60, fine) == 0 && calls == 0);       // less than what is set
  CHECK(limit.raise(2, 200, fine) == 0 && calls == 1);      // more, on this device alone
  CHECK(limit.raise(3, 100, fine) == 0 && calls == 1);
  CHECK(limit.raise(5, 100, [] { return 7; }) == 7);        // a failure is handed on and tried again
  CHECK(limit.raise(5, 100, fine) == 0 && calls == 2);
  for (int dev : {-1, tllm::PerDeviceLimit::DEVICES}) {     // no place for these: set at every call
    CHECK(limit.raise(dev, 1, fine) == 0 && limit.raise(dev, 1, fine) == 0);
  }
  CHECK(calls == 6);
  std::atomic<int> at_once{0};
  std::vector<std::thread> threads;
  for (int i = 0; i < 8; ++i)
    threads.emplace_back([&] { for (int dev = 8; dev < 40; ++dev) limit.raise(dev, 10, [&] { ++at_once; return 0; }); });
  for (auto& t : threads) t.join();
  CHECK(at_once == 32);
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_a_limit_is_raised_once_on_every_device(tmp_path):
    src, exe = tmp_path / "per_device.cpp", tmp_path / "per_device"
    src.write_text(PER_DEVICE)
    res = subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", build.CSRC, "-o", str(exe), str(src)], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    assert subprocess.run([str(exe)], timeout=60).returncode == 0      # else the line of the check


def test_every_launch_raises_its_shared_memory_per_device():
    """cudaFuncSetAttribute holds for the current device only: it is called in one place, which keeps a limit per device."""
    where = {name: text.count("cudaFuncSetAttribute(") for name, text in sources().items()}
    assert {n: c for n, c in where.items() if c} == {"common.cuh": 1}


def test_every_wait_that_gives_up_has_a_code_and_words_of_its_own():
    from tiny_llm_b200 import ops
    codes, reports = {}, {}
    for name, text in sources().items():
        for role, code in re.findall(r"\b(ERR_[A-Z_]+) = (\d+)", text):
            assert name == "tc_common.cuh", f"{role} of {name}: the codes are kept in one list"
            codes[role] = int(code)
        for role in re.findall(r"atomicExch\([^;]*?(\w+)\)", text):
            reports.setdefault(role, set()).add(name)
    assert len(set(codes.values())) == len(codes) and 0 not in codes.values()
    assert set(reports) == set(codes)
    assert all(len(files) == 1 for files in reports.values())          # no two kernel families share a code
    assert set(ops._STATUS_CODES) == set(codes.values()) and len(set(ops._STATUS_CODES.values())) == len(codes)
    with pytest.raises(ops.KernelError, match=rf"code {codes['ERR_DR_CONSUMER']}: .*scan"):
        ops.raise_status("cuda:63", codes["ERR_DR_CONSUMER"])
    with pytest.raises(ops.KernelError, match=rf"code {codes['ERR_SK_PRODUCER']}: .*32-bit product"):
        ops.raise_status("cuda:63", codes["ERR_SK_PRODUCER"])


# kernels whose copies to shared memory complete on an mbarrier
STREAMED = ["linear_generic.cu"]


@pytest.mark.parametrize("name", STREAMED)
def test_a_producer_that_gives_up_waits_for_its_copies(name):
    """Every kernel that arms a barrier with the bytes of a copy ends its producer with the wait for the copies in flight."""
    kernels = [k for k in sources()[name].split("__global__")[1:] if "mbar_expect_tx(" in k]
    assert kernels and all("mbar_drain(" in k for k in kernels)


ROUTE = r"""
#include "attention_route.h"
#include <cstdio>
// tokens, longest, requests, keys, nq, nk, values -> rows per CTA
int main() {
  long long t, q, r, k;
  int nq, nk, d;
  while (std::scanf("%lld %lld %lld %lld %d %d %d", &t, &q, &r, &k, &nq, &nk, &d) == 7)
    std::printf("%d ", tllm::attention_rows_per_cta(t, q, r, k, nq, nk, d > 64, 148));
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_rows_share_a_cta_only_where_that_was_measured_to_be_no_slower(tmp_path):
    src, exe = tmp_path / "route.cpp", tmp_path / "route"
    src.write_text(ROUTE)
    res = subprocess.run(["g++", "-std=c++17", "-I", build.CSRC, "-o", str(exe), str(src)], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    cases = [
        # decoded tokens of groups of four and more, prompts, portions behind a context
        ((8, 1, 8, 700, 32, 4, 64), 4), ((8, 1, 0, 0, 32, 4, 64), 4), ((1, 1, 1, 300, 16, 4, 64), 4),
        ((509, 509, 1, 509, 32, 4, 64), 16), ((60, 60, 1, 60, 32, 32, 128), 4), ((7, 7, 1, 1507, 32, 32, 128), 4),
        ((4, 4, 1, 1504, 28, 4, 128), 4), ((64, 1, 64, 255, 32, 4, 64), 4), ((33, 33, 1, 33, 20, 4, 64), 4),
        # a head with keys of its own, decoded: nothing is shared
        ((8, 1, 8, 2000, 32, 32, 128), 0), ((3, 3, 1, 900, 16, 16, 64), 0),
        # few keys
        ((8, 1, 8, 9, 32, 4, 64), 0), ((4, 4, 1, 4, 32, 4, 64), 0), ((17, 17, 1, 17, 32, 32, 128), 0), ((64, 1, 64, 31, 32, 4, 64), 0),
        # few requests whose tokens would be walked one after the other, and many of them
        ((4, 1, 4, 700, 28, 4, 128), 0), ((24, 20, 5, 700, 32, 32, 128), 0), ((20, 4, 17, 1400, 32, 32, 128), 0),
        ((24, 20, 5, 700, 12, 4, 64), 0), ((24, 20, 0, 700, 12, 4, 64), 0), ((16, 1, 16, 40, 28, 4, 128), 0),
        ((16, 1, 16, 700, 28, 4, 128), 4), ((67, 4, 64, 1400, 8, 4, 64), 4), ((67, 4, 64, 1400, 32, 32, 128), 4),
        # portions of several requests: each brings more rows than a CTA takes
        ((72, 24, 3, 24, 12, 4, 64), 4), ((30, 10, 3, 900, 32, 32, 128), 4),
    ]
    text = "\n".join(" ".join(map(str, c)) for c, _ in cases)
    got = subprocess.run([str(exe)], input=text, capture_output=True, text=True, timeout=60).stdout.split()
    assert [int(g) for g in got] == [want for _, want in cases]
