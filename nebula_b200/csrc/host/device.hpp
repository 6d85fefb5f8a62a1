// Device-side helpers shared by the host implementation files: status
// checks, owning device buffers, and the device copies of geometry and
// materials.
#pragma once
#include <cuda_runtime.h>
#include <vector>
#include <string>
#include <algorithm>
#include <cmath>
#include <limits>
#include "internal.hpp"
#include "../kernels.cuh"

namespace nbl {

#define CU(call)                                                                          \
	do {                                                                                  \
		cudaError_t e_ = (call);                                                          \
		if (e_ != cudaSuccess)                                                            \
			throw Error(e_ == cudaErrorMemoryAllocation ? NBL_ERR_OOM : NBL_ERR_CUDA,     \
				std::string(#call) + ": " + cudaGetErrorString(e_));                     \
	} while (0)

inline void set_device(int device)
{
	int n = 0;
	if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0)
		throw Error(NBL_ERR_NO_DEVICE, "no CUDA device available");
	require(device >= 0 && device < n, "device ordinal out of range");
	CU(cudaSetDevice(device));
}

// Device buffer that frees itself.
struct DevBuf {
	void* p = nullptr;
	size_t bytes = 0;
	DevBuf() = default;
	explicit DevBuf(size_t n) { alloc(n); }
	void alloc(size_t n)
	{
		release();
		if (n == 0) return;
		CU(cudaMalloc(&p, n));
		bytes = n;
	}
	void release()
	{
		if (p) cudaFree(p);
		p = nullptr;
		bytes = 0;
	}
	~DevBuf() { release(); }
	DevBuf(const DevBuf&) = delete;
	DevBuf& operator=(const DevBuf&) = delete;
	template<class T> T* as() const { return static_cast<T*>(p); }
};

// A triangle in the 48-byte device layout.
inline DevTriangle device_triangle(const nbl_triangle& t)
{
	DevTriangle d;
	d.r0x = t.r0[0]; d.r0y = t.r0[1]; d.r0z = t.r0[2]; d.mat_in = t.material_in;
	d.e1x = t.e1[0]; d.e1y = t.e1[1]; d.e1z = t.e1[2]; d.mat_out = t.material_out;
	d.e2x = t.e2[0]; d.e2y = t.e2[1]; d.e2z = t.e2[2]; d.pad0 = 0;
	return d;
}

// A triangle's plane in units of what rounding can shift it by.
//
// The ray test (intersect_ray) returns t = num / det with, for a ray from s
// along d, det = -d.n + a, num = (s - r0).n + b, where n = e1 x e2 and the
// rounding of the two cross and dot products (u = 2^-24 per operation) gives
// |a| <= 8 u |d| |e1| |e2| and |b| <= 10 u |s - r0| |e1| |e2|.  With H the
// height of r0's plane over s along n, times |n|, and S = d.n, t lies in
// (0, L] only if H sgn(S) >= -(|b| + 2 |a| L) and |H| <= L (|S| + |a|) + |b|
// (if |S| <= |a| the sign of t is open, but then |t| > L for an |H| larger
// than |b| + 2 |a| L).  L |d| is at most the domain's diagonal D, so both
// allowances are at most 26 u (|s - r0| + D) |e1| |e2| / |n| as a distance;
// evaluating the plane in float adds at most 16 u times the largest
// coordinate.  The unit below is larger than their sum.
inline DevPlane plane_of(const nbl_triangle& t, const HostGeometry& g)
{
	const double u = 1.0 / (1 << 24);
	double e1[3], e2[3], r0[3], n[3], far = 0, coord = 0, aa = 0, bb = 0, nn = 0;
	for (int k = 0; k < 3; ++k) {
		e1[k] = t.e1[k]; e2[k] = t.e2[k]; r0[k] = t.r0[k];
		const double reach = std::fabs(r0[k] - g.center[k]) + g.halfsize[k];
		far += reach * reach;
		coord = std::max(coord, std::max(std::fabs(r0[k]), std::fabs((double)g.center[k]) + g.halfsize[k]));
		aa += e1[k] * e1[k];
		bb += e2[k] * e2[k];
	}
	for (int k = 0; k < 3; ++k) {
		n[k] = e1[(k + 1) % 3] * e2[(k + 2) % 3] - e1[(k + 2) % 3] * e2[(k + 1) % 3];
		nn += n[k] * n[k];
	}
	const double len = std::sqrt(nn);
	const double unit = 32 * u * ((std::sqrt(far) + g.max_extent) * std::sqrt(aa * bb) / len + 2 * coord);
	const double w = (n[0] * r0[0] + n[1] * r0[1] + n[2] * r0[2]) / len / unit;
	DevPlane p;
	p.x = (float)(n[0] / len / unit); p.y = (float)(n[1] / len / unit); p.z = (float)(n[2] / len / unit);
	p.w = (float)w;
	if (!(len > 0) || !std::isfinite(unit) || !std::isfinite(w))
		p.x = p.y = p.z = p.w = std::numeric_limits<float>::quiet_NaN();
	return p;
}

// Whether a mesh is fine in the sense of PASS_EMPTY: its leaves are small
// against the flights, so that most of those crossed hold no triangle.
inline bool fine_mesh(const HostGeometry& g) { return g.octree.size() >= (size_t)1 << 20; }

// Geometry resident on one device.
struct DeviceGeometry {
	DevBuf octree, tris, planes;
	DevGeometry view{};
	void upload(const HostGeometry& g, cudaStream_t s)
	{
		std::vector<DevTriangle> dt(g.tris.size());
		std::vector<DevPlane> dp(g.tris.size());
		for (size_t i = 0; i < g.tris.size(); ++i) {
			dt[i] = device_triangle(g.tris[i]);
			dp[i] = plane_of(g.tris[i], g);
		}
		octree.alloc(g.octree.size() * sizeof(int32_t));
		tris.alloc(std::max<size_t>(dt.size(), 1) * sizeof(DevTriangle));
		planes.alloc(std::max<size_t>(dp.size(), 1) * sizeof(DevPlane));
		CU(cudaMemcpyAsync(octree.p, g.octree.data(), g.octree.size() * sizeof(int32_t), cudaMemcpyHostToDevice, s));
		if (!dt.empty()) {
			CU(cudaMemcpyAsync(tris.p, dt.data(), dt.size() * sizeof(DevTriangle), cudaMemcpyHostToDevice, s));
			CU(cudaMemcpyAsync(planes.p, dp.data(), dp.size() * sizeof(DevPlane), cudaMemcpyHostToDevice, s));
		}
		CU(cudaStreamSynchronize(s));
		view.octree = octree.as<int32_t>();
		view.tris = tris.as<DevTriangle>();
		view.planes = planes.as<DevPlane>();
		view.cx = g.center[0]; view.cy = g.center[1]; view.cz = g.center[2];
		view.hx = g.halfsize[0]; view.hy = g.halfsize[1]; view.hz = g.halfsize[2];
		view.max_extent = g.max_extent;
		view.n_tri = (int32_t)g.tris.size();
		view.n_octree = (int64_t)g.octree.size();
	}
};

// Materials resident on one device: one buffer of all tables plus the
// DevMaterial array pointing into it.
struct DeviceMaterials {
	DevBuf tables, mats;
	int n = 0;
	std::vector<DevMaterial> host;   // the device array's contents
	void upload(const std::vector<const HostMaterial*>& ms, cudaStream_t s, uint32_t phys = PH_DEFAULT)
	{
		const bool kieft = (phys & PH_KIEFT) != 0;
		n = (int)ms.size();
		std::vector<float> blob;
		std::vector<size_t> offs;
		auto add = [&](const HostTable& t) {
			size_t o = blob.size();
			o = (o + 31) & ~size_t(31);   // 128-byte aligned tables
			blob.resize(o);
			offs.push_back(o);
			blob.insert(blob.end(), t.data.begin(), t.data.end());
		};
		for (const HostMaterial* m : ms) {
			const InelasticTables it = inelastic_tables(*m, kieft);
			add(m->el_imfp); add(m->el_icdf); add(*it.imfp); add(*it.omega); add(*it.q); add(*it.binding);
		}
		tables.alloc(std::max<size_t>(blob.size(), 1) * sizeof(float));
		CU(cudaMemcpyAsync(tables.p, blob.data(), blob.size() * sizeof(float), cudaMemcpyHostToDevice, s));
		std::vector<DevMaterial> dm(ms.size());
		const float* base = tables.as<float>();
		size_t k = 0;
		auto dev = [&](const HostTable& t) {
			DevTable d;
			d.data = base + offs[k++];
			d.nx = t.nx; d.ny = t.ny; d.nz = t.nz; d.pad = 0;
			d.x_min = t.x_min; d.x_step = t.x_step; d.y_min = t.y_min; d.y_step = t.y_step;
			d.z_min = t.z_min; d.z_step = t.z_step;
			return d;
		};
		for (size_t i = 0; i < ms.size(); ++i) {
			const HostMaterial& m = *ms[i];
			DevMaterial& d = dm[i];
			const InelasticTables it = inelastic_tables(m, kieft);
			d.el_imfp = dev(m.el_imfp); d.el_icdf = dev(m.el_icdf); d.in_imfp = dev(*it.imfp);
			d.in_omega = dev(*it.omega); d.in_q = dev(*it.q); d.in_binding = dev(*it.binding);
			d.fermi = m.fermi; d.band_gap = m.band_gap; d.barrier = m.barrier;
			d.phonon_loss = m.phonon_loss; d.recoil_const = m.recoil_const;
			d.in_scale = 1.0f; d.el_scale = 1.0f; d.pad = 0;
		}
		mats.alloc(std::max<size_t>(dm.size(), 1) * sizeof(DevMaterial));
		CU(cudaMemcpyAsync(mats.p, dm.data(), dm.size() * sizeof(DevMaterial), cudaMemcpyHostToDevice, s));
		CU(cudaStreamSynchronize(s));
		host = dm;
	}
};

}  // namespace nbl
