"""The staged copy of pageable memory (csrc/host/pageable.hpp) on the host.

The header is compiled against stand-ins for the CUDA calls it makes, which
copy with memcpy and fail where a case asks for it: the copy is complete for
sizes at the edges of its blocks, and a set-up that fails (page-locked memory,
events, threads, memory for threads) leaves the caller with the direct copy or
the copy's own thread, never with an error or an aborted process.
"""
import os
import subprocess

import pytest

from nebula_b200 import build

PROGRAM = r"""
#include "host/pageable.hpp"
#include <atomic>
#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <string>
#include <vector>
#include <pthread.h>

static std::string fail;
static int countdown = -1;              // operator new fails when it reaches zero
static std::atomic<int> events{0}, synced{0}, last_error{0};

void* operator new(size_t n)
{
	if (countdown >= 0 && countdown-- == 0) throw std::bad_alloc();
	if (void* p = std::malloc(n ? n : 1)) return p;
	throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

static cudaError_t set(cudaError_t e) { last_error = e; return e; }
extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
{
	if (fail == "buffer") return set(cudaErrorMemoryAllocation);
	*p = std::malloc(n);
	return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned)
{
	if (fail == "event" && events >= 3) return set(cudaErrorMemoryAllocation);
	++events;
	*e = (cudaEvent_t)std::malloc(1);
	return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { --events; std::free(e); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { ++synced; return cudaSuccess; }
cudaError_t cudaGetLastError() { return (cudaError_t)last_error.exchange(0); }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t)
{
	if (fail == "copy") return cudaErrorInvalidValue;
	std::memcpy(d, s, n);
	return cudaSuccess;
}
#ifdef NO_THREADS
int pthread_create(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*) { return EAGAIN; }
#endif
}

int main(int argc, char** argv)
{
	const size_t n = std::strtoull(argv[1], nullptr, 10);
	fail = argc > 2 ? argv[2] : "";
	std::vector<unsigned char> src(n), dst(n + 1, 0xEE);
	unsigned x = 1;
	for (auto& b : src) b = (unsigned char)((x = x * 1664525u + 1013904223u) >> 24);
	{
		nbl::PageableCopy c;
		const bool made = c.make();
		if (made == (fail == "buffer" || fail == "event")) return 2;
		if (last_error != 0) return 3;                // a failure's error does not stay behind
		if (!made) {                                  // a later try succeeds
			fail = "";
			if (!c.make()) return 4;
		}
		nbl::PageableCopy d;                          // a copy of FIRST_BYTES makes the buffers
		if (d.takes(c.MIN_BYTES - 1) || d.takes(c.MIN_BYTES - 1)) return 9;
		if (!d.takes(c.FIRST_BYTES) || !d.takes(c.MIN_BYTES) || d.takes(c.MIN_BYTES - 1)) return 10;
		nbl::PageableCopy w;                          // of smaller ones the second asks for them
		for (int k = 0; k < 2; ++k) {
			if (w.make_wanted(), w.takes(c.MIN_BYTES)) return 11;
			if (w.takes(c.MIN_BYTES - 1)) return 12;
		}
		if (w.make_wanted(), !w.takes(c.MIN_BYTES)) return 13;
		// the second helper thread finds no memory, after the first has started
		if (fail == "memory") countdown = 1;
		const cudaError_t e = c.run(dst.data(), src.data(), n, 0, nullptr);
		countdown = -1;
		if (fail == "copy") return e == cudaErrorInvalidValue && synced == 1 ? 0 : 5;
		if (e != cudaSuccess) return 6;
	}
	if (events != 0) return 7;
	if (std::memcmp(dst.data(), src.data(), n) != 0 || dst[n] != 0xEE) return 8;
	return 0;
}
"""


@pytest.fixture(scope="module")
def programs(tmp_path_factory):
    d = tmp_path_factory.mktemp("pageable")
    src = d / "copy.cpp"
    src.write_text(PROGRAM)
    out = {}
    for name, defs in (("threads", []), ("no_threads", ["-DNO_THREADS"])):
        out[name] = str(d / name)
        subprocess.run(["g++", "-std=c++17", "-O1", "-I" + build.CSRC, "-I" + os.path.join(build.CUDA_HOME, "include")]
                       + defs + [str(src), "-o", out[name], "-pthread"], check=True)
    return out


BLOCK = 256 << 10


@pytest.mark.parametrize("n", [1, BLOCK - 1, BLOCK, BLOCK + 1, 4 * BLOCK, 8 * BLOCK + 1, (16 << 20) + 36])
@pytest.mark.parametrize("program", ["threads", "no_threads"])
def test_copies_every_byte(programs, program, n):
    assert subprocess.run([programs[program], str(n)], timeout=60).returncode == 0


@pytest.mark.parametrize("fail", ["buffer", "event", "memory", "copy"])
def test_failed_setup_or_copy(programs, fail):
    assert subprocess.run([programs["threads"], str((16 << 20) + 36), fail], timeout=60).returncode == 0
