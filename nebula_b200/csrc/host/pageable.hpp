// Host to device copies of pageable memory through several threads.
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <cstddef>
#include <cstring>
#include <thread>

namespace nbl {

// The driver stages a pageable copy through one thread (10 to 12 GB/s); here
// four threads copy blocks of it into page-locked buffers and send them on from
// there (21 GB/s).  Making the buffers takes some 3.5 ms, which a copy has to
// earn before it is faster than the driver's: B200, direct / first copy with
// the buffers / later ones, in ms: 33 MB 2.2 / 4.3 / 1.7, 64 MB 4.9 / 6.3 / 3.1,
// 80 MB 6.9 / 7.1 / 3.8, 92 MB 8.2 / 7.7 / 4.3, 256 MB 23 / 15.3 / 11.8.  (Of the
// block sizes 128 KiB gives 6.3 ms for 92 MB and 1 MiB 3.6, but the larger the
// buffers the longer they take to make.)
class PageableCopy {
public:
	// from here on a simulation's first copy is no slower than the driver's
	static constexpr size_t MIN_BYTES = (size_t)80 << 20;
	static constexpr int LANES = 4;
	static constexpr size_t BLOCK = (size_t)256 << 10;

	PageableCopy() = default;
	PageableCopy(const PageableCopy&) = delete;
	PageableCopy& operator=(const PageableCopy&) = delete;
	~PageableCopy()
	{
		for (Lane& l : lanes)
			for (cudaEvent_t e : l.sent)
				if (e) cudaEventDestroy(e);
		if (buffer) cudaFreeHost(buffer);
	}

	// Makes the buffers, once.  False where that is not possible: such a copy
	// is the driver's, which needs none of them.
	bool make()
	{
		bool made = buffer || cudaHostAlloc((void**)&buffer, 2 * LANES * BLOCK, cudaHostAllocDefault) == cudaSuccess;
		for (Lane& l : lanes)
			for (cudaEvent_t& e : l.sent)
				made = made && (e || cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess);
		if (!made)
			cudaGetLastError();
		return made;
	}

	// Enqueues on `stream` (of the current device, `device`) and returns when
	// all of it has arrived.  make() has returned true before.
	cudaError_t run(void* dst, const void* src, size_t bytes, int device, cudaStream_t stream)
	{
		const auto part = [=](int lane) { work(lane, dst, src, bytes, device, stream); };
		std::thread helpers[LANES - 1];
		int started = 0;
		try {
			for (; started < LANES - 1; ++started)
				helpers[started] = std::thread(part, started + 1);
		} catch (...) {
			// no more threads (or no memory for them): their blocks are copied
			// here; those that started are joined below
		}
		part(0);
		for (int i = started + 1; i < LANES; ++i)
			part(i);
		for (int i = 0; i < started; ++i)
			helpers[i].join();
		const cudaError_t e = cudaStreamSynchronize(stream);
		for (const Lane& l : lanes)
			if (l.err != cudaSuccess)
				return l.err;
		return e;
	}

private:
	struct Lane {
		cudaEvent_t sent[2] = { nullptr, nullptr };
		cudaError_t err = cudaSuccess;
	};
	Lane lanes[LANES];
	char* buffer = nullptr;       // 2 MiB

	// blocks lane, lane + LANES, ... through the lane's two buffers in turn
	void work(int lane, void* dst, const void* src, size_t bytes, int device, cudaStream_t stream) noexcept
	{
		Lane& l = lanes[lane];
		l.err = cudaSetDevice(device);
		int turn = 0;
		for (size_t at = (size_t)lane * BLOCK; at < bytes && l.err == cudaSuccess; at += LANES * BLOCK, turn ^= 1) {
			const size_t n = std::min(BLOCK, bytes - at);
			char* const b = buffer + (2 * lane + turn) * BLOCK;
			// the buffer's last block has left it (no record yet: nothing to wait for)
			l.err = cudaEventSynchronize(l.sent[turn]);
			if (l.err != cudaSuccess) break;
			std::memcpy(b, static_cast<const char*>(src) + at, n);
			l.err = cudaMemcpyAsync(static_cast<char*>(dst) + at, b, n, cudaMemcpyHostToDevice, stream);
			if (l.err != cudaSuccess) break;
			l.err = cudaEventRecord(l.sent[turn], stream);
		}
	}
};

}  // namespace nbl
