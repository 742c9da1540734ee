"""The exact k-NN's kept device memory (``csrc/scratch.cuh``), compiled for the host with a stand-in for the
GPU's allocator: a thread that calls on several devices gets memory of the device that it calls on."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "hnsw_engine_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <map>
#include <thread>
#include "scratch.cuh"

static int current = 0;
static bool full = false;
static std::map<void *, int> owner;  // live blocks and their device

struct FakeMem {
    static bool device(int *d) { *d = current; return true; }
    static bool alloc(void **p, size_t bytes) {
        if (full) return false;
        *p = new char[bytes];
        owner[*p] = current;
        return true;
    }
    static void release(int d, void *p) {
        if (owner.at(p) != d) std::printf("block of device %d released on %d\n", owner.at(p), d);
        owner.erase(p);
        delete[] static_cast<char *>(p);
    }
};

#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)

int main() {
    int rc = 0;
    std::thread([&] {
        rc = [] {
            static thread_local DeviceScratch<FakeMem> s;
            void *a = s.get(1000);
            CHECK(a && owner.at(a) == 0);
            CHECK(s.get(400) == a);                       // kept
            current = 1;
            void *b = s.get(400);                         // smaller, another device
            CHECK(b && b != a && owner.at(b) == 1);
            current = 0;
            CHECK(s.get(1000) == a);                      // the first device's is still there
            void *c = s.get(5000);                        // grows where it is
            CHECK(c && owner.at(c) == 0 && owner.size() == 2);
            full = true;
            CHECK(s.get(9000) == nullptr);
            full = false;
            CHECK(owner.size() == 1 && s.get(9000) != nullptr);
            current = 64;
            CHECK(s.get(1) == nullptr);
            current = 3;
            return 0;
        }();
    }).join();
    CHECK(rc == 0);
    CHECK(owner.empty());                                 // a thread's end gives back every device's
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host compiler")
def test_each_device_has_its_own_block(tmp_path: Path) -> None:
    src, exe = tmp_path / "scratch_test.cpp", tmp_path / "scratch_test"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0 and run.stdout == "", run.stdout
