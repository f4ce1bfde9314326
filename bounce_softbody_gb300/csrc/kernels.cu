// Single-body kernels other than the solve (solve.cu): elements, row assembly, contact filter,
// state transfer, ray casts.
#include "device.cuh"
#include "ops.h"

#include <cstdlib>
#include <cstring>

#include <algorithm>

namespace b3g {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

int grid_for(int items, int per_block)
{
	int g = (items + per_block - 1) / per_block;
	if (g < 1) g = 1;
	if (g > kMaxPartials) g = kMaxPartials;
	return g;
}

// ------------------------------------------------------------------ kernels
// A later Newton iteration of a step whose Newton loop already ended: its kernels do nothing.
__device__ __forceinline__ bool newton_over(const DevBody& B, const StepParams& P)
{
	return !P.first_newton && B.sc->newton_done;
}

__global__ void __launch_bounds__(kThreads) k_tets(DevBody B, StepParams P)
{
	if (newton_over(B, P)) return;
	for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < B.nt; e += gridDim.x * blockDim.x) tet_element(B, e, P);
}

__global__ void __launch_bounds__(kThreads) k_tris(DevBody B, StepParams P)
{
	if (newton_over(B, P)) return;
	for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < B.ntr; e += gridDim.x * blockDim.x) tri_element(B, e, P);
}

__global__ void __launch_bounds__(kThreads) k_springs(DevBody B, StepParams P)
{
	if (newton_over(B, P)) return;
	for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < B.ns; e += gridDim.x * blockDim.x) spring_element(B, e, P);
}

// stretch/shear triangles and mouse springs in one launch: the triangles, then the springs
__global__ void __launch_bounds__(kThreads) k_cloth_forces(DevBody B, StepParams P)
{
	if (newton_over(B, P)) return;
	const int total = B.nbw + B.nms;
	for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x)
	{
		if (e < B.nbw) bw_element(B, e, P);
		else mouse_element(B, e - B.nbw, P);
	}
}

// ------------------------------------------------------------------ ray casts
// b3TriangleShape::RayCast (triangle_shape.cpp:314-387) for the segment p1 + t d, t in [0, 1].
// Returns the fraction and the plane offset num = n . (A - p1), whose sign orients the normal.
__device__ __forceinline__ bool ray_triangle(float3 p1, float3 d, float3 A, float3 B, float3 C, float& t, float& num,
                                             float3& n)
{
	if (dot3(d, d) < kFltEps * kFltEps) return false;
	const float3 AB = B - A, AC = C - A;
	n = normalize3(cross3(AB, AC));
	num = dot3(n, A - p1);
	const float den = dot3(n, d);
	if (den == 0.0f) return false;
	t = num / den;
	if (t < 0.0f || 1.0f < t) return false;
	const float3 Q = p1 + t * d;
	const float3 QA = A - Q, QB = B - Q, QC = C - Q;
	const float3 N = cross3(AB, AC);
	const float u = dot3(cross3(QB, QC), N);
	const float v = dot3(cross3(QC, QA), N);
	const float w = dot3(cross3(QA, QB), N);
	return u >= 0.0f && v >= 0.0f && w >= 0.0f;
}

__device__ __forceinline__ unsigned long long ray_key(float t, unsigned tri)
{
	// a hit has 0 <= t <= 1, and non-negative floats order like their bit patterns; fmaxf maps
	// -0 (which passes the t < 0 test) to +0
	return ((unsigned long long)__float_as_uint(fmaxf(t, 0.0f)) << 32) | tri;
}

// grid.x strides over triangles, grid.y over segments; one 64-bit atomicMin per warp and segment
__global__ void __launch_bounds__(kThreads) k_ray_cast(DevBody B, int ntri, const float* __restrict__ seg,
                                                        unsigned count, unsigned long long* keys)
{
	const int lane = threadIdx.x & 31;
	for (unsigned r = blockIdx.y; r < count; r += gridDim.y)
	{
		const float3 p1 = f3(seg[6 * r], seg[6 * r + 1], seg[6 * r + 2]);
		const float3 d = f3(seg[6 * r + 3], seg[6 * r + 4], seg[6 * r + 5]) - p1;
		const int stride = gridDim.x * blockDim.x;
		for (int base = blockIdx.x * blockDim.x; base < ntri; base += stride)
		{
			const int e = base + threadIdx.x;
			unsigned long long key = ~0ull;
			if (e < ntri)
			{
				const uint4 id = B.tri[e];
				float t, num;
				float3 n;
				if (ray_triangle(p1, d, ld3(B.x, id.x), ld3(B.x, id.y), ld3(B.x, id.z), t, num, n))
					key = ray_key(t, (unsigned)e);
			}
#pragma unroll
			for (int o = 16; o > 0; o >>= 1)
			{
				const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o);
				key = other < key ? other : key;
			}
			if (lane == 0 && key != ~0ull) atomicMin(keys + r, key);
		}
	}
}

// A segment's hit from its key: the winner's normal, oriented as the reference orients it.
__device__ __forceinline__ b3g_ray_hit ray_hit(const DevBody& B, float3 p1, float3 d, unsigned long long key)
{
	b3g_ray_hit o;
	o.hit = 0;
	o.triangle = 0;
	o.fraction = 0.0f;
	o.normal[0] = o.normal[1] = o.normal[2] = 0.0f;
	if (key != ~0ull)
	{
		const unsigned e = (unsigned)(key & 0xffffffffu);
		const uint4 id = B.tri[e];
		float t, num;
		float3 n;
		ray_triangle(p1, d, ld3(B.x, id.x), ld3(B.x, id.y), ld3(B.x, id.z), t, num, n);
		if (num > 0.0f) n = -n;
		o.hit = 1;
		o.triangle = e;
		o.fraction = __uint_as_float((unsigned)(key >> 32));
		o.normal[0] = n.x;
		o.normal[1] = n.y;
		o.normal[2] = n.z;
	}
	return o;
}

// One thread per segment
__global__ void k_ray_finish(DevBody B, const float* __restrict__ seg, unsigned count,
                             const unsigned long long* __restrict__ keys, b3g_ray_hit* hits)
{
	const unsigned r = blockIdx.x * blockDim.x + threadIdx.x;
	if (r >= count) return;
	const float3 p1 = f3(seg[6 * r], seg[6 * r + 1], seg[6 * r + 2]);
	hits[r] = ray_hit(B, p1, f3(seg[6 * r + 3], seg[6 * r + 4], seg[6 * r + 5]) - p1, keys[r]);
}

// A few segments in one launch: they come in the kernel's parameters, the last CTA of a segment writes
// its hit, and keys (kept inverted, so that zero is "no hit yet") and arrival counters are left at
// zero for the next call. A pick is all latency: a copy, a memset, two launches and a copy back
// took 45 us a call from Python for 8 segments on 18432 triangles, the kernels 9 of them.
__global__ void __launch_bounds__(kThreads) k_ray_pick(DevBody B, int ntri, RaySegments S, RayScratch* w, b3g_ray_hit* hits)
{
	const int lane = threadIdx.x & 31, r = blockIdx.y;
	const float* seg = S.s[r];
	const float3 p1 = f3(seg[0], seg[1], seg[2]);
	const float3 d = f3(seg[3], seg[4], seg[5]) - p1;
	unsigned long long best = 0ull;
	for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < ntri; e += gridDim.x * blockDim.x)
	{
		const uint4 id = B.tri[e];
		float t, num;
		float3 n;
		if (ray_triangle(p1, d, ld3(B.x, id.x), ld3(B.x, id.y), ld3(B.x, id.z), t, num, n))
		{
			const unsigned long long key = ~ray_key(t, (unsigned)e);
			best = key > best ? key : best;
		}
	}
#pragma unroll
	for (int o = 16; o > 0; o >>= 1)
	{
		const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
		best = other > best ? other : best;
	}
	if (lane == 0 && best) atomicMax(&w->key[r], best);
	__syncthreads();
	if (threadIdx.x != 0) return;
	__threadfence();
	if (atomicAdd(&w->arrived[r], 1u) != gridDim.x - 1) return;
	__threadfence();
	const unsigned long long key = ~atomicExch(&w->key[r], 0ull);
	w->arrived[r] = 0u;
	hits[r] = ray_hit(B, p1, d, key);
}

// Filtered contacts: the contact update and each vertex's constraint at the start of a step
__global__ void __launch_bounds__(kThreads) k_contact_filter(DevBody B, float h)
{
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < B.n; i += gridDim.x * blockDim.x)
		contact_filter_vertex(B, i, h);
}

template <class TA, class TV, bool FILTER>
__global__ void __launch_bounds__(kThreads) k_assemble(DevBody B, StepParams P, int init)
{
	if (newton_over(B, P)) return;
	// the grid team's reduction memory starts at zero
	for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < (int)(sizeof(TeamMemory) / 4); k += gridDim.x * blockDim.x)
		((unsigned*)B.team)[k] = 0u;
	if (blockIdx.x == 0 && threadIdx.x == 0) solve_pending(B, P.first_newton);
	const int lane = threadIdx.x & 31;
	for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < B.nslices; s += (gridDim.x * blockDim.x) >> 5)
		assemble_row<TA, TV, LdPlain, FILTER>(B, s, lane, P, init);
}

// The row assembly of a small body, one CTA per slice: a warp per slot column (slot k of the slice's 32
// rows) and one for the rows' right-hand sides and vertex terms, where k_assemble has one warp do them
// in turn. A small body leaves most of the GPU idle, and a row's slots are a chain of dependent
// gathers: 10^3 block 50 us with one warp a slice (4 CTAs). Every block and right-hand side is summed in
// k_assemble's order.
constexpr int kSlotWarps = 17;

template <class TA, class TV>
__global__ void __launch_bounds__(32 * kSlotWarps) k_assemble_slots(DevBody B, StepParams P, int init)
{
	if (newton_over(B, P)) return;
	for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < (int)(sizeof(TeamMemory) / 4); k += gridDim.x * blockDim.x)
		((unsigned*)B.team)[k] = 0u;
	if (blockIdx.x == 0 && threadIdx.x == 0) solve_pending(B, P.first_newton);
	__shared__ float sb[3][32], sk[9][32], sd[32];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, slots = (int)(blockDim.x >> 5) - 1;
	const int i = blockIdx.x * kSlice + lane;
	const bool row = i < B.n;
	const bool Si = row && B.type[i] == B3G_DYNAMIC;
	const int base = B.slice_ptr[blockIdx.x];
	const int w = row ? B.rowlen[i] : 0;
	float a[9];
	if (warp == slots)
	{
		if (row)
		{
			float extra, Kc[9];
			const float3 bi = row_vertex_terms<LdPlain, false, false>(B, i, P, Si, extra, Kc);
			sb[0][lane] = bi.x;
			sb[1][lane] = bi.y;
			sb[2][lane] = bi.z;
			sd[lane] = extra;
#pragma unroll
			for (int q = 0; q < 9; ++q) sk[q][lane] = Kc[q];
		}
	}
	else
	{
		// a later column than the diagonal of warp 0 comes first, so that the diagonal stays in a
		for (int k = warp + (B.maxw - 1 - warp) / slots * slots; k >= 0; k -= slots)
		{
			if (k >= w) continue;
			slot_block<LdPlain>(B, base + k * kSlice + lane, a);
			if (k == 0) break;
			const size_t bs = block_slot((size_t)base, k, lane);
			if (!(Si && B.type[B.col[bs]] == B3G_DYNAMIC))
			{
#pragma unroll
				for (int q = 0; q < 9; ++q) a[q] = 0.0f;
			}
			store_block<TA>(B, bs, a);
		}
	}
	__syncthreads();
	if (warp != 0 || !row) return;
#pragma unroll
	for (int q = 0; q < 9; ++q) a[q] += P.h * P.h * sk[q][lane];
	a[0] += sd[lane];
	a[4] += sd[lane];
	a[8] += sd[lane];
	float3 bi = f3(sb[0][lane], sb[1][lane], sb[2][lane]);
	if (!Si)
	{
#pragma unroll
		for (int q = 0; q < 9; ++q) a[q] = (q == 0 || q == 4 || q == 8) ? 1.0f : 0.0f;
		bi = f3(0, 0, 0);
	}
	store_block<TA>(B, block_slot((size_t)base, 0, lane), a);
	row_finish<TV>(B, i, bi, a, init);
}

__global__ void __launch_bounds__(kThreads) k_nostep(DevBody B)
{
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < B.n; i += gridDim.x * blockDim.x)
	{
		float3 x = ld3(B.x, i);
		if (B.contacts)
			for (int k = 0; k < B.nw; ++k)
			{
				const int c = i * B.nw + k;
				if (B.c_exists[c] && (B.type[i] != B3G_DYNAMIC || !aabb_overlap(x, B.srad[i], B.shapes[k]))) B.c_exists[c] = 0;
				else if (B.c_exists[c])
				{
					B.c_nf[c] = 0.0f;
					B.c_apply[c] = 0;
				}
			}
		st3(B.fext, i, f3(0, 0, 0));
		st3(B.trans, i, f3(0, 0, 0));
		if (B.contacts) find_new_contacts(B, i, x);
	}
}

__global__ void k_accumulate(float* dst, const float* src, size_t n)
{
	for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) dst[i] += src[i];
}

// b3Particle::SetType (particle.cpp:58-87) for every vertex whose type changes: external force
// and translation cleared, velocity zeroed for static vertices, contacts destroyed.
__global__ void k_set_types(DevBody B, const int8_t* nt)
{
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < B.n; i += gridDim.x * blockDim.x)
	{
		int8_t t = nt[i];
		if (t == B.type[i]) continue;
		st3(B.fext, i, f3(0, 0, 0));
		st3(B.trans, i, f3(0, 0, 0));
		if (t == B3G_STATIC) st3(B.v, i, f3(0, 0, 0));
		for (int k = 0; k < B.nw; ++k) B.c_exists[i * B.nw + k] = 0;
		((int8_t*)B.type)[i] = t;
	}
}

__global__ void k_fill(float* p, size_t n, float v)
{
	for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) p[i] = v;
}

// Bodies up to this many slices are assembled by k_assemble_slots (6 CTAs per SM). Measured with
// k_assemble / k_assemble_slots, us a step: 378 vertices with three Newton iterations 707 / 644, 10^3
// block 206 / 186, FP64 block of 397 slices 615 / 573, cloth of 512 slices 1257 / 1240; blocks of 2229 and 8192
// slices, which fill the GPU with a warp a slice, 3431 / 3544 and 11491 / 11673.
constexpr int kSlotAssemblySlices = 1024;

StepParams dev_params(const StepParamsHost& P)
{
	StepParams p;
	p.h = P.h;
	p.first_newton = P.first_newton;
	return p;
}

int slice_grid(const DevBody& B) { return grid_for(B.nslices, kWarps); }

// Grid of the per-vertex kernels (contact filter, steps without a solve, types): at most two CTAs
// per SM, each thread striding over several vertices. B3G_VERTEX_CTAS overrides the cap (read once).
int vertex_grid(const DevBody& B)
{
	static const int cap = [] {
		const char* e = std::getenv("B3G_VERTEX_CTAS");
		if (e) return std::atoi(e);
		int dev = 0, sms = 0;
		cudaGetDevice(&dev);
		cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
		return 2 * sms;
	}();
	const int g = grid_for(B.n, kThreads);
	return cap > 0 && cap < g ? cap : g;
}

} // namespace

// CTAs over the triangles: enough to fill the GPU for one segment, fewer per segment when there are
// many segments
static int ray_ctas(int ntri, uint32_t count)
{
	static const int sms = [] {
		int dev = 0, n = 0;
		cudaGetDevice(&dev);
		cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
		return n > 0 ? n : 1;
	}();
	return std::max(1, std::min(grid_for(ntri, kThreads), 4 * sms / (int)std::min<uint32_t>(count, 64)));
}

cudaError_t op_ray_cast(const DevBody& B, int ntri, const float* segments, uint32_t count, unsigned long long* keys,
                        b3g_ray_hit* hits, cudaStream_t st)
{
	if (count == 0) return cudaSuccess;
	cudaError_t e = cudaMemsetAsync(keys, 0xff, count * sizeof(unsigned long long), st);
	if (e != cudaSuccess) return e;
	if (ntri > 0)
	{
		const int per_seg = ray_ctas(ntri, count);
		dim3 grid((unsigned)per_seg, std::min<uint32_t>(count, 65535u));
		k_ray_cast<<<grid, kThreads, 0, st>>>(B, ntri, segments, count, keys);
	}
	k_ray_finish<<<(count + 127) / 128, 128, 0, st>>>(B, segments, count, keys, hits);
	return cudaGetLastError();
}

cudaError_t op_ray_pick(const DevBody& B, int ntri, const float* segments, uint32_t count, RayScratch* scratch,
                        b3g_ray_hit* hits, cudaStream_t st)
{
	if (count == 0) return cudaSuccess;
	RaySegments S;
	std::memcpy(S.s, segments, 6 * sizeof(float) * (size_t)count);
	const dim3 grid((unsigned)ray_ctas(ntri, count), count);
	k_ray_pick<<<grid, kThreads, 0, st>>>(B, ntri, S, scratch, hits);
	return cudaGetLastError();
}

cudaError_t op_elements(const DevBody& B, const StepParamsHost& Ph, cudaStream_t st)
{
	StepParams P = dev_params(Ph);
	if (B.nt > 0) k_tets<<<grid_for(B.nt, kThreads), kThreads, 0, st>>>(B, P);
	if (B.ntr > 0) k_tris<<<grid_for(B.ntr, kThreads), kThreads, 0, st>>>(B, P);
	if (B.ns > 0) k_springs<<<grid_for(B.ns, kThreads), kThreads, 0, st>>>(B, P);
	if (B.nbw + B.nms > 0) k_cloth_forces<<<grid_for(B.nbw + B.nms, kThreads), kThreads, 0, st>>>(B, P);
	return cudaGetLastError();
}

cudaError_t op_assemble(const DevBody& B, const StepParamsHost& Ph, int prec, int init, cudaStream_t st)
{
	StepParams P = dev_params(Ph);
	int g = slice_grid(B);
	const int in = init;
	if (B.filt)
	{
		if (prec == kP64) k_assemble<double, double, true><<<g, kThreads, 0, st>>>(B, P, in);
		else if (prec == kPBF) k_assemble<__nv_bfloat16, float, true><<<g, kThreads, 0, st>>>(B, P, in);
		else k_assemble<float, float, true><<<g, kThreads, 0, st>>>(B, P, in);
	}
	else if (B.nslices <= kSlotAssemblySlices)
	{
		const int t = 32 * std::min(kSlotWarps, B.maxw + 1);
		if (prec == kP64) k_assemble_slots<double, double><<<B.nslices, t, 0, st>>>(B, P, in);
		else if (prec == kPBF) k_assemble_slots<__nv_bfloat16, float><<<B.nslices, t, 0, st>>>(B, P, in);
		else k_assemble_slots<float, float><<<B.nslices, t, 0, st>>>(B, P, in);
	}
	else if (prec == kP64) k_assemble<double, double, false><<<g, kThreads, 0, st>>>(B, P, in);
	else if (prec == kPBF) k_assemble<__nv_bfloat16, float, false><<<g, kThreads, 0, st>>>(B, P, in);
	else k_assemble<float, float, false><<<g, kThreads, 0, st>>>(B, P, in);
	return cudaGetLastError();
}

cudaError_t op_contact_filter(const DevBody& B, float h, cudaStream_t st)
{
	k_contact_filter<<<vertex_grid(B), kThreads, 0, st>>>(B, h);
	return cudaGetLastError();
}

cudaError_t op_nostep(const DevBody& B, cudaStream_t st)
{
	k_nostep<<<vertex_grid(B), kThreads, 0, st>>>(B);
	return cudaGetLastError();
}

// grid.y walks the bodies, grid.x (with a stride) the floats of one body
__global__ void __launch_bounds__(kThreads) k_batch_scatter_add(const XferBody* __restrict__ table, unsigned count,
                                                                 const float* __restrict__ src)
{
	for (unsigned b = blockIdx.y; b < count; b += gridDim.y)
	{
		const XferBody t = table[b];
		const float* s = src + t.off;
		for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < t.n3; k += gridDim.x * blockDim.x)
			t.fext[k] += s[k];
	}
}

__global__ void __launch_bounds__(kThreads) k_batch_gather(const XferBody* __restrict__ table, unsigned count,
                                                            float* __restrict__ dx, float* __restrict__ dv)
{
	for (unsigned b = blockIdx.y; b < count; b += gridDim.y)
	{
		const XferBody t = table[b];
		for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < t.n3; k += gridDim.x * blockDim.x)
		{
			if (dx) dx[t.off + k] = t.x[k];
			if (dv) dv[t.off + k] = t.v[k];
		}
	}
}

static dim3 xfer_grid(uint32_t count, uint32_t max_n3)
{
	return dim3((unsigned)std::max(1u, std::min<uint32_t>((max_n3 + kThreads - 1) / kThreads, 64u)),
	            std::min<uint32_t>(std::max(count, 1u), 65535u));
}

cudaError_t op_batch_scatter_add(const XferBody* table, uint32_t count, uint32_t max_n3, const float* src,
                                 cudaStream_t st)
{
	if (count == 0) return cudaSuccess;
	k_batch_scatter_add<<<xfer_grid(count, max_n3), kThreads, 0, st>>>(table, count, src);
	return cudaGetLastError();
}

cudaError_t op_batch_gather(const XferBody* table, uint32_t count, uint32_t max_n3, float* dst_x, float* dst_v,
                            cudaStream_t st)
{
	if (count == 0) return cudaSuccess;
	k_batch_gather<<<xfer_grid(count, max_n3), kThreads, 0, st>>>(table, count, dst_x, dst_v);
	return cudaGetLastError();
}

cudaError_t op_accumulate(float* dst, const float* src, size_t count, cudaStream_t st)
{
	if (count == 0) return cudaSuccess;
	int g = (int)((count + kThreads - 1) / kThreads);
	if (g > 4096) g = 4096;
	k_accumulate<<<g, kThreads, 0, st>>>(dst, src, count);
	return cudaGetLastError();
}

cudaError_t op_set_types(const DevBody& B, const int8_t* new_types, cudaStream_t st)
{
	k_set_types<<<vertex_grid(B), kThreads, 0, st>>>(B, new_types);
	return cudaGetLastError();
}

cudaError_t op_fill_f32(float* p, size_t count, float value, cudaStream_t st)
{
	if (count == 0) return cudaSuccess;
	int g = (int)((count + kThreads - 1) / kThreads);
	if (g > 4096) g = 4096;
	k_fill<<<g, kThreads, 0, st>>>(p, count, value);
	return cudaGetLastError();
}

} // namespace b3g
