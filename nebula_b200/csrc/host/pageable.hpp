// Host to device copies of pageable memory through several threads.
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <cstddef>
#include <cstring>
#include <thread>

namespace nbl {

// The driver stages a pageable copy through one thread (10 to 12 GB/s); here four
// threads copy blocks of it into page-locked buffers and send them on from there
// (21 GB/s).  Making the buffers takes some 3 ms, which a copy has to earn before
// it is faster than the driver's: B200, direct / first copy with the buffers made
// for it / later ones, in ms: 17 MB 1.2 / 3.5 / 1.0, 25 MB 1.7 / 3.7 / 1.35, 33
// MB 2.3 / 4.3 / 1.8, 48 MB 3.4 / 5.6 / 2.4, 64 MB 4.9 / 6.3 / 3.1, 80 MB 6.9 /
// 7.1 / 3.8, 92 MB 7.9 / 7.7 / 4.4, 256 MB 23 / 15.3 / 11.8.  So a copy of
// FIRST_BYTES makes the buffers at once.  Of those from MIN_BYTES on the first
// two are the driver's: an object that copies a second time is likely to go on,
// and the buffers are made where the host next waits for the device
// (nbl_sim::advance).  (Of the block sizes 128 KiB gives 5.8 ms for 92 MB and 64
// KiB 8.6: each block's copy takes 8 us to issue.  1 MiB gives 3.6, but the
// larger the buffers the longer they take to make.)
class PageableCopy {
public:
	static constexpr size_t MIN_BYTES = (size_t)24 << 20;
	static constexpr size_t FIRST_BYTES = (size_t)80 << 20;
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

	// Whether this copy of pageable memory should go through run().  False: it
	// is the driver's, which needs no buffers.
	bool takes(size_t bytes)
	{
		if (bytes < MIN_BYTES)
			return false;
		if (!ready && bytes >= FIRST_BYTES)
			make();
		wanted = again && !ready;
		again = true;
		return ready;
	}

	// Makes the buffers if a copy would have liked them.
	void make_wanted()
	{
		if (wanted)
			make();
		wanted = false;
	}

	// Makes the buffers, once.  False where that is not possible.
	bool make()
	{
		bool made = buffer || cudaHostAlloc((void**)&buffer, 2 * LANES * BLOCK, cudaHostAllocDefault) == cudaSuccess;
		for (Lane& l : lanes)
			for (cudaEvent_t& e : l.sent)
				made = made && (e || cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess);
		if (!made)
			cudaGetLastError();
		ready = made;
		return made;
	}

	// Enqueues on `stream` (of the current device, `device`) and returns when
	// all of it has arrived.  make() or takes() has returned true before.
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
	bool ready = false;           // it and the events are made
	bool again = false;           // there was a copy of MIN_BYTES
	bool wanted = false;          // there was another, without the buffers

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
