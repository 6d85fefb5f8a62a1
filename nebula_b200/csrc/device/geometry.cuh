// Octree ray walk and ray-triangle test, bit-exact with the reference CPU
// build on identical float32 inputs.
//
// The walk visits the same leaf cells in the same order as
// octree<gpu_flag>::propagate (reference geometry/octree.inl:33-192), because
// the returned distance accumulates float roundoff along that exact cell
// sequence.  Every float operation is written as an explicitly rounded
// intrinsic (__fadd_rn, __fmul_rn, __fdiv_rn ...), so the compiler can neither
// contract a multiply-add into an FMA nor reorder: the result equals the
// x86-64 SSE evaluation of the reference's expressions, which is what the
// parity tests check.
//
// What is B200-specific is the data path: triangles are 48-byte records read
// with three 128-bit read-only loads, their planes 16-byte records in an array
// of their own, and the node array is read through the read-only cache; the
// whole structure stays L2-resident for the workloads of interest.
#pragma once
#include "../nbl_device_types.h"

namespace nbl {

__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fs(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fd(float a, float b) { return __fdiv_rn(a, b); }

// dot(a, b) = a.x*b.x + a.y*b.y + a.z*b.z evaluated left to right
// (reference common/vector_math.h:107-110)
__device__ __forceinline__ float dot3(float ax, float ay, float az, float bx, float by, float bz)
{
	return fa(fa(fm(ax, bx), fm(ay, by)), fm(az, bz));
}

// 10 * FLT_EPSILON (reference config/data_types.h:58)
#define NBL_EPS (10.0f * 1.1920928955078125e-07f)

struct TriHit { float t; };

// Moller-Trumbore as triangle::intersect_ray (reference core/triangle.inl:7-28):
// -1 on miss.  The reference divides before it compares; a numerator that
// misses its bound by more than the quotient's rounding is rejected by a
// multiplication first, and the three divisions are left to the triangles that
// are hit (1 in 5 of those tested) and to borderline ones.
__device__ __forceinline__ float intersect_ray(const DevTriangle& T, float sx, float sy, float sz,
	float dx, float dy, float dz)
{
	// pvec = cross(dir, e2)
	const float px = fs(fm(dy, T.e2z), fm(dz, T.e2y));
	const float py = fs(fm(dz, T.e2x), fm(dx, T.e2z));
	const float pz = fs(fm(dx, T.e2y), fm(dy, T.e2x));
	const float det = dot3(T.e1x, T.e1y, T.e1z, px, py, pz);
	const float size = fabsf(det);
	if (size < NBL_EPS)
		return -1.0f;
	const float tx = fs(sx, T.r0x), ty = fs(sy, T.r0y), tz = fs(sz, T.r0z);
	const float un = dot3(tx, ty, tz, px, py, pz);
	const float us = det < 0.0f ? -un : un;
	if ((us < -1.01f * NBL_EPS * size) || (us > 1.001f * size))
		return -1.0f;
	// qvec = cross(start - r0, e1)
	const float qx = fs(fm(ty, T.e1z), fm(tz, T.e1y));
	const float qy = fs(fm(tz, T.e1x), fm(tx, T.e1z));
	const float qz = fs(fm(tx, T.e1y), fm(ty, T.e1x));
	const float vn = dot3(dx, dy, dz, qx, qy, qz);
	const float vs = det < 0.0f ? -vn : vn;
	if ((vs < -1.01f * NBL_EPS * size) || (us + vs > 1.001f * size))
		return -1.0f;
	const float u = fd(un, det);
	if ((u < -NBL_EPS) || (u > 1.0f + NBL_EPS))
		return -1.0f;
	const float v = fd(vn, det);
	if ((v < -NBL_EPS) || (fa(u, v) > 1.0f + NBL_EPS))
		return -1.0f;
	const float t = fd(dot3(T.e2x, T.e2y, T.e2z, qx, qy, qz), det);
	if (t < 0.0f)
		return -1.0f;
	return t;
}

__device__ __forceinline__ DevTriangle load_tri(const DevTriangle* __restrict__ tris, int i)
{
	const float4* p = reinterpret_cast<const float4*>(tris + i);
	const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
	DevTriangle t;
	t.r0x = a.x; t.r0y = a.y; t.r0z = a.z; t.mat_in = __float_as_int(a.w);
	t.e1x = b.x; t.e1y = b.y; t.e1z = b.z; t.mat_out = __float_as_int(b.w);
	t.e2x = c.x; t.e2y = c.y; t.e2z = c.z; t.pad0 = 0;
	return t;
}

// The triangle's normal, cross(e1, e2) with the float operations of
// triangle::get_normal (reference core/triangle.inl:75-78).
__device__ __forceinline__ void tri_normal(const DevTriangle& T, float& nx, float& ny, float& nz)
{
	nx = fs(fm(T.e1y, T.e2z), fm(T.e1z, T.e2y));
	ny = fs(fm(T.e1z, T.e2x), fm(T.e1x, T.e2z));
	nz = fs(fm(T.e1x, T.e2y), fm(T.e1y, T.e2x));
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
__device__ __forceinline__ DevPlane plane_of(const DevTriangle& T, const DevGeometry& g)
{
	const double u = 1.0 / (1 << 24);
	const double e1[3] = { T.e1x, T.e1y, T.e1z }, e2[3] = { T.e2x, T.e2y, T.e2z }, r0[3] = { T.r0x, T.r0y, T.r0z };
	const double center[3] = { g.cx, g.cy, g.cz }, half[3] = { g.hx, g.hy, g.hz };
	double n[3], far = 0, coord = 0, aa = 0, bb = 0, nn = 0;
#pragma unroll
	for (int k = 0; k < 3; ++k) {
		const double reach = fabs(r0[k] - center[k]) + half[k];
		far += reach * reach;
		coord = fmax(coord, fmax(fabs(r0[k]), fabs(center[k]) + half[k]));
		aa += e1[k] * e1[k];
		bb += e2[k] * e2[k];
	}
#pragma unroll
	for (int k = 0; k < 3; ++k) {
		n[k] = e1[(k + 1) % 3] * e2[(k + 2) % 3] - e1[(k + 2) % 3] * e2[(k + 1) % 3];
		nn += n[k] * n[k];
	}
	const double len = sqrt(nn);
	const double unit = 32 * u * ((sqrt(far) + g.max_extent) * sqrt(aa * bb) / len + 2 * coord);
	const double w = (n[0] * r0[0] + n[1] * r0[1] + n[2] * r0[2]) / len / unit;
	DevPlane p;
	p.x = (float)(n[0] / len / unit); p.y = (float)(n[1] / len / unit); p.z = (float)(n[2] / len / unit);
	p.w = (float)w;
	if (!(len > 0) || !isfinite(unit) || !isfinite(w))
		p.x = p.y = p.z = p.w = __int_as_float(0x7fffffff);
	return p;
}

// Whether the ray test could return a distance in (0, limit] for the triangle
// with plane `pl`: false only when its rounded result provably lies outside,
// because the ray meets the plane behind the start or past `limit` by more
// than the rounding (1 in the plane's units).  Any NaN keeps the triangle.
__device__ __forceinline__ bool plane_in_reach(const DevPlane& pl, float sx, float sy, float sz, float dx, float dy,
	float dz, float limit)
{
	const float h = __fmaf_rn(-pl.z, sz, __fmaf_rn(-pl.y, sy, __fmaf_rn(-pl.x, sx, pl.w)));
	const float s = __fmaf_rn(pl.z, dz, __fmaf_rn(pl.y, dy, fm(pl.x, dx)));
	const float ahead = s < 0.0f ? -h : h;
	return !(ahead < -1.0f) && !(ahead > __fmaf_rn(fabsf(s), limit, 1.0f));
}

__device__ __forceinline__ DevPlane load_plane(const DevPlane* __restrict__ planes, int i)
{
	const float4 a = __ldg(reinterpret_cast<const float4*>(planes + i));
	DevPlane p;
	p.x = a.x; p.y = a.y; p.z = a.z; p.w = a.w;
	return p;
}

// octree::in_domain (reference geometry/octree.inl:25-30)
__device__ __forceinline__ bool in_domain(const DevGeometry& g, float x, float y, float z)
{
	return (x > fs(g.cx, g.hx)) && (x < fa(g.cx, g.hx)) && (y > fs(g.cy, g.hy)) && (y < fa(g.cy, g.hy))
		&& (z > fs(g.cz, g.hz)) && (z < fa(g.cz, g.hz));
}

// Where a walk stands between leaf cells: the current point, the distance
// left, the location code of the cell it is about to enter and the cells
// walked so far.  A walk cut short after some cells resumes from this state
// with exactly the float values it would have carried on with.
struct WalkState {
	float cx, cy, cz, to_go;
	uint64_t location;
	int steps;
};

__device__ __forceinline__ WalkState walk_start(float sx, float sy, float sz, float distance)
{
	WalkState w;
	w.cx = sx; w.cy = sy; w.cz = sz; w.to_go = distance;
	w.location = 1;
	w.steps = 0;
	return w;
}

// Status of a walk that stopped at its cell budget (propagate_cells).
#define NBL_WALK_PENDING (-3)

// Nearest triangle hit within `distance` along a (normalised) direction,
// ignoring `ignore_tri` and triangles whose outgoing material equals
// `ignore_mat`, walking from state `w` (walk_start for a new walk).  Returns
// the triangle index (or -1) and the distance (or `distance` itself when
// nothing is hit).  A walk longer than `max_steps` leaf cells in all stops
// early and reports -2 (the host counts these as errors; the reference has no
// such bound).  With `max_cells` > 0, a walk that has not ended after
// `max_cells` cells in this call returns NBL_WALK_PENDING with `w` holding
// where it stands; calling again with that state continues the same cell
// sequence with the same float values.  Before each cell of that budget up to
// `pass_empty` leaves without triangles are passed (they cost a descent each).
// `bounded`: the walk starts inside the
// root cell, which the planes' rounding units are made for (every transport
// flight does); without it every listed triangle gets the full test.
__device__ __forceinline__ int propagate_cells(const DevGeometry& g, WalkState& w,
	float dx, float dy, float dz, float distance, int ignore_tri, int ignore_mat, float& out_dist,
	int max_cells = 0, int pass_empty = 0, int max_steps = 1 << 20, bool bounded = true)
{
	const int32_t* __restrict__ od = g.octree;
	float cx = w.cx, cy = w.cy, cz = w.cz;
	float to_go = w.to_go;
	uint64_t location = w.location;
	int steps = w.steps;
	int cells = 0;
	// to the next cell: move to the exit face, then neighbour cell by
	// location-code arithmetic
	const auto advance = [&](float intersect, int face) {
		to_go = fs(to_go, intersect);
		cx = fa(cx, fm(dx, intersect));
		cy = fa(cy, fm(dy, intersect));
		cz = fa(cz, fm(dz, intersect));
		const unsigned int mask = (unsigned int)(-face);
		unsigned int value;
		if (mask == 1u) value = (dx >= 0.0f) ? 0u : 1u;
		else if (mask == 2u) value = (dy >= 0.0f) ? 0u : 2u;
		else value = (dz >= 0.0f) ? 0u : 4u;
#pragma unroll 1
		while (location > 1) {
			if ((location & mask) == value) {
				location ^= mask;
				break;
			}
			location >>= 3;
		}
		++steps;
	};
	const auto pending = [&]() {
		w.cx = cx; w.cy = cy; w.cz = cz; w.to_go = to_go;
		w.location = location;
		w.steps = steps;
		out_dist = distance;
		return NBL_WALK_PENDING;
	};
	out_dist = distance;
	do {
		float intersect;
		int target, index, entry;
		// up to `pass_empty` leaves without triangles come along with the next cell
#pragma unroll 1
		for (int empty = 0; ; ++empty) {
			// Cell centre update of the reference, c += (aw * h) * (bit - 0.5)
			// with aw = 2^-level: both products are exact (power-of-two
			// scalings of h, far from underflow), so the offset is carried as
			// +-h 2^-(level+1), halved per level, and only the addition rounds.
			float ax = g.cx, ay = g.cy, az = g.cz, aw = 1.0f;
			float ox = fm(g.hx, 0.5f), oy = fm(g.hy, 0.5f), oz = fm(g.hz, 0.5f);
			index = 0;
			// descend to the current location code from the root
#pragma unroll 1
			for (int i = 60 - __clzll((long long)location); i >= 0; i -= 3) {
				const unsigned int octant = (unsigned int)(location >> i) & 7u;
				index = __ldg(od + index + octant);
				ax = fa(ax, (octant & 1u) ? ox : -ox);
				ay = fa(ay, (octant & 2u) ? oy : -oy);
				az = fa(az, (octant & 4u) ? oz : -oz);
				aw = fm(aw, 0.5f);
				ox = fm(ox, 0.5f); oy = fm(oy, 0.5f); oz = fm(oz, 0.5f);
			}
			// continue to the leaf that contains the current position
#pragma unroll 1
			while (index >= 0) {
				const bool bx = cx > ax, by = cy > ay, bz = cz > az;
				const unsigned int octant = (bx ? 1u : 0u) | (by ? 2u : 0u) | (bz ? 4u : 0u);
				location = (location << 3) | octant;
				index = __ldg(od + index + octant);
				ax = fa(ax, bx ? ox : -ox);
				ay = fa(ay, by ? oy : -oy);
				az = fa(az, bz ? oz : -oz);
				aw = fm(aw, 0.5f);
				ox = fm(ox, 0.5f); oy = fm(oy, 0.5f); oz = fm(oz, 0.5f);
			}
			index = -index;

			// exit distance through the leaf's faces (AABB_intersect, octree.inl:212-220)
			{
				const float hx = fm(aw, g.hx), hy = fm(aw, g.hy), hz = fm(aw, g.hz);
				const float tx = fd(fs(fa(ax, copysignf(fa(hx, NBL_EPS), dx)), cx), dx);
				const float ty = fd(fs(fa(ay, copysignf(fa(hy, NBL_EPS), dy)), cy), dy);
				const float tz = fd(fs(fa(az, copysignf(fa(hz, NBL_EPS), dz)), cz), dz);
				if ((tx < ty) && (tx < tz)) { intersect = tx; target = -1; }
				else if ((ty < tx) && (ty < tz)) { intersect = ty; target = -2; }
				else { intersect = tz; target = -4; }
			}

			entry = __ldg(od + index);
			if (entry >= 0 || empty == pass_empty)
				break;
			if (intersect >= to_go)
				return -1;
			advance(intersect, target);
			if (steps > max_steps)
				return -2;
			if (location <= 1)
				return -1;
		}

		// Triangles of the leaf, in two passes of up to 32 list entries.  The
		// first marks those whose plane the ray can meet within the distance
		// that matters: a hit past the cell's exit or the distance left
		// changes nothing, except that hits within NBL_EPS of one another
		// replace each other in list order, which moves the accepted distance
		// up by at most NBL_EPS per list entry (4096 are allowed for).  The
		// second tests the marked ones in list order.  The full test costs
		// several times the plane's, few triangles need it, and a warp's
		// second loop is as long as its lane with the most marked triangles
		// instead of the longest list: 3 654 instructions per 32 electrons on
		// the grating against 4 212 with one pass and the full test for every
		// entry (kernel 68.5 / 75.7 ms, 160 x 160 x 100 primaries).
		const float limit = fa(fminf(intersect, to_go), 4096.0f * NBL_EPS);
#pragma unroll 1
		for (; entry >= 0; index += 32) {
			unsigned marked = 0u;
			int k = 0;
#pragma unroll 1
			do {
				const DevPlane pl = load_plane(g.planes, entry);
				const int next = __ldg(od + index + k + 1);
				if (entry != ignore_tri && (!bounded || plane_in_reach(pl, cx, cy, cz, dx, dy, dz, limit)))
					marked |= 1u << k;
				entry = next;
				++k;
			} while (entry >= 0 && k < 32);
#pragma unroll 1
			for (; marked; marked &= marked - 1u) {
				const int ti = __ldg(od + index + __ffs(marked) - 1);
				const DevTriangle T = load_tri(g.tris, ti);
				const float t = intersect_ray(T, cx, cy, cz, dx, dy, dz);
				if ((t > 0.0f) && (t <= fa(intersect, NBL_EPS))) {
					// (the material test comes first in the reference; few
					// triangles are left for it here)
					float nx, ny, nz;
					tri_normal(T, nx, ny, nz);
					const int mat_out = dot3(nx, ny, nz, dx, dy, dz) < 0.0f ? T.mat_in : T.mat_out;
					if (mat_out != ignore_mat) {
						intersect = t;
						target = ti;
					}
				}
			}
		}

		if (intersect >= to_go)
			return -1;
		if (target >= 0) {
			out_dist = fa(fs(distance, to_go), intersect);
			return target;
		}
		advance(intersect, target);
		if (steps > max_steps)
			return -2;
		if (++cells == max_cells && location > 1)
			return pending();
	} while (location > 1);
	return -1;
}

// The whole walk in one call (octree<gpu_flag>::propagate).
__device__ __forceinline__ int propagate(const DevGeometry& g, float sx, float sy, float sz,
	float dx, float dy, float dz, float distance, int ignore_tri, int ignore_mat, float& out_dist,
	int max_steps = 1 << 20)
{
	WalkState w = walk_start(sx, sy, sz, distance);
	return propagate_cells(g, w, dx, dy, dz, distance, ignore_tri, ignore_mat, out_dist, 0, 0, max_steps,
		in_domain(g, sx, sy, sz));
}

}  // namespace nbl
