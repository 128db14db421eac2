"""Grants of shared memory (csrc/grant.h) against a runtime that only counts: compiled for the host, no GPU and no CUDA library."""
import os
import re
import subprocess

import pytest

from bitnet_c_b200.csrc import build

PROGRAM = r"""
#include "grant.h"
#include <cstdio>
#include <thread>
#include <vector>
static thread_local int device = 0;
static int asked[100], last[100], fail = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int bytes) {
  if (fail) return cudaErrorInvalidValue;
  ++asked[device];
  last[device] = bytes;
  return cudaSuccess;
}
#define CHECK(x) if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; }
static BnGrant grant, other;
int main() {
  CHECK(grant.ask(nullptr, 47 * 1024, 1024) == cudaSuccess && asked[0] == 0);      // no grant needed
  CHECK(other.ask(nullptr, 47 * 1024, 1025) == cudaSuccess && asked[0] == 1);  // with what the kernel has beside it, one is
  asked[0] = 0;
  fail = 1;
  CHECK(grant.ask(nullptr, 100 * 1024, 1024) == cudaErrorInvalidValue);
  fail = 0;
  CHECK(grant.ask(nullptr, 100 * 1024, 1024) == cudaSuccess && asked[0] == 1);     // what failed is not taken for granted
  CHECK(grant.ask(nullptr, 60 * 1024, 1024) == cudaSuccess && asked[0] == 1 && last[0] == 100 * 1024);  // never less
  CHECK(other.ask(nullptr, 60 * 1024, 1024) == cudaSuccess && asked[0] == 2);      // another kernel
  device = 1;
  CHECK(grant.ask(nullptr, 60 * 1024, 1024) == cudaSuccess && asked[1] == 1 && last[1] == 60 * 1024);  // another device
  CHECK(grant.ask(nullptr, 120 * 1024, 1024) == cudaSuccess && asked[1] == 2 && last[1] == 120 * 1024);
  device = 70;
  CHECK(grant.ask(nullptr, 60 * 1024, 1024) == cudaSuccess && grant.ask(nullptr, 60 * 1024, 1024) == cudaSuccess && asked[70] == 2);
  std::vector<std::thread> threads;
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([t] {
      device = 2;
      for (int i = 0; i < 1000; ++i) grant.ask(nullptr, (50 + (i * 7 + t) % 100) * 1024, 0);
    });
  for (auto& t : threads) t.join();
  CHECK(last[2] == 149 * 1024 && asked[2] <= 100);
  return 0;
}
"""


def test_shared_memory_is_granted_per_device(tmp_path):
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.find_nvcc())), "include")
    (tmp_path / "grant.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "grant")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-pthread", "-I", os.path.dirname(build.__file__), "-I", cuda,
                    str(tmp_path / "grant.cpp"), "-o", exe], check=True, timeout=300)
    p = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert p.returncode == 0, p.stdout


@pytest.mark.parametrize("family", ["linear", "sampling", "attention", "moe_few"])
def test_kernels_that_once_needed_no_grant_ask_per_device(family):
    """Products of few rows in float32, nucleus sampling, attention and experts of few tokens ran on a second device of a process
    without any grant; one flag for all devices left their kernels without it there."""
    with open(os.path.join(os.path.dirname(build.__file__), build.SOURCES[family])) as f:
        assert "static bool granted" not in f.read()


@pytest.mark.parametrize("family", sorted(build.SOURCES))
def test_no_kernel_has_two_grants(family):
    """A macro with a grant of its own that is written out twice for the same kernel leaves it with two, of which one lowers what the other
    relies on."""
    with open(os.path.join(os.path.dirname(build.__file__), build.SOURCES[family])) as f:
        text = f.read().replace("\\\n", " ")
    for name in re.findall(r"#define (\w+)\([^)]*\)[^\n]*static BnGrant", text):
        for line in re.findall(r"#define (\w+)\(([^)]*)\)([^\n]*)", text):
            if name + "(" in line[2]:  # written out by another macro: count that one's arguments through
                outer, params, body = line
                inner = re.findall(rf"\b{name}\(([^)]*)\)", body)
                text += "\n" + "\n".join(f"{name}({_put(i, params, args)})" for args in re.findall(rf"(?<!define )\b{outer}\(([^)]*)\)", text) for i in inner)
        made = [a for line in text.split("\n") if "#define" not in line for a in re.findall(rf"\b{name}\(([^)]*)\)", line)]
        assert made and len(made) == len(set(made)), (name, sorted(made))


def _put(args, params, values):
    given = dict(zip((p.strip() for p in params.split(",")), (v.strip() for v in values.split(","))))
    return ", ".join(given.get(a.strip(), a.strip()) for a in args.split(","))
