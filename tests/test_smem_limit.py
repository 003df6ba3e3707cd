"""-m "not gpu": dynamic shared memory above 48 KB is asked for once per device and kernel (csrc/launch.h: allow_smem), against a stand-in for the
CUDA runtime with two devices; no launcher keeps that per process."""
import glob
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "yalm_b200", "csrc")

PROGRAM = r"""
#include "launch.h"
#include <cstdio>
#include <thread>
static thread_local int current = 0;
static std::mutex mu;
static std::map<std::pair<int, const void *>, int> limit; // what each device would have
static int calls = 0, fail = 0;
extern "C" cudaError_t cudaGetDevice(int *d) { return *d = current, cudaSuccess; }
extern "C" cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 1, cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute, int v) {
	std::lock_guard<std::mutex> lock(mu);
	++calls;
	if (fail) return cudaErrorInvalidValue;
	limit[{current, f}] = v;
	return cudaSuccess;
}
extern "C" cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *, int, size_t) { return *n = 1, cudaSuccess; }
static void kernel_a() {}
static void kernel_b() {}
#define CHECK(x) \
	if (!(x)) return std::printf("%s\n", #x), 1
int main() {
	const void *a = (const void *)kernel_a, *b = (const void *)kernel_b;
	cudaError_t err;
	CHECK(yalm::allow_smem(a, 48 * 1024) == cudaSuccess && calls == 0);
	for (int dev = 0; dev < 2; ++dev) {
		current = dev, calls = 0;
		CHECK(yalm::allow_smem(a, 100000) == cudaSuccess && (limit[{dev, a}] == 100000));
		CHECK(yalm::allow_smem(a, 60000) == cudaSuccess && (limit[{dev, a}] == 100000) && calls == 1); // never lowered, not asked again
		CHECK(yalm::resident_ctas(b, 256, 70000, &err) == 1 && err == cudaSuccess && (limit[{dev, b}] == 70000));
	}
	fail = 1;
	CHECK(yalm::allow_smem(a, 200000) == cudaErrorInvalidValue);
	fail = 0;
	CHECK(yalm::allow_smem(a, 200000) == cudaSuccess && (limit[{1, a}] == 200000)); // a refusal is not kept
	std::thread t[8]; // each device's first callers at once
	limit.clear();
	int bad = 0;
	for (int i = 0; i < 8; ++i)
		t[i] = std::thread([&, i] {
			current = 2 + i % 4;
			bool ok = yalm::allow_smem(a, 90000) == cudaSuccess;
			std::lock_guard<std::mutex> lock(mu);
			if (!ok || limit[{current, a}] != 90000) ++bad; // (before its own launch)
		});
	for (auto &x : t) x.join();
	CHECK(bad == 0);
	return 0;
}
"""


def test_each_device_is_asked(tmp_path):
    src, exe = tmp_path / "limit.cpp", tmp_path / "limit"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-I", os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"),
                           str(src), "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_no_launcher_keeps_it_per_process():
    for path in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")):
        assert not re.search(r"static\s+(bool|size_t)\s+configured\s*=", open(path).read()), path
