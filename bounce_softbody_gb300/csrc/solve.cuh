// The PCG of one body as one cooperative launch over the whole GPU (the grid team).
//
// What bounds it: a body's matrix is a few MB, so an iteration moves it in microseconds; what the
// earlier launches per iteration paid for was launch latency, a reduction through one counter, and
// the solver vectors' round trips. Here the whole solve is one launch. A CTA owns a contiguous run
// of 32-row slices for the launch: their vectors (r, d, q, x, and the scalar Jacobi) stay in shared
// memory, and so does as much of their matrix as fits; only s, which neighbours gather, goes
// through global memory (L2). Besides s, two team-wide sums per iteration are all that is exchanged:
// d.q after q = A s + beta q, d = s + beta d, and r.s after r -= alpha q, s = M^-1 r. x += alpha d
// runs while the second sum is on its way.
//
// Team sums. Every CTA stores its partial in its slot as two words, mantissa and exponent (Fixed), each
// with two bits of the sum's number; one warp of every CTA polls all slots and adds them up, so every
// thread holds the same bits and takes the same decisions. No fence and no atomic is on that path. Above
// 16 CTAs the slots exist 16 times, a replica for every 16th CTA: with one copy the pollers' traffic on
// the same lines costs 0.4 / 1.4 / 3.8 us a sum for 4 / 32 / 152 CTAs, with sixteen 0.9 / 0.95 / 1.6
// (slots of one word). Two slot arrays alternate: a CTA can only overwrite its slot of sum e with that
// of sum e + 2 after every CTA has arrived at sum e + 1, and so has read sum e. The same holds for s,
// rewritten only after the sum that follows the sweep which gathers it.
// s itself needs no barrier in the FP32 and BF16 modes on small bodies: its fourth component carries the
// number of its version, a vertex's 16 bytes are written and read as one access at GPU scope, and a
// gather that meets an older version reads again. What does not fit one access (FP64 vectors, x of a
// refresh), and the s that a large body gathers through the L1, is published by a fence of one of the
// CTA's warps and a flag behind it that the team polls with the sum's slots: the fence alone costs 900
// clocks, most of them beside the sum and the update of x.
// All polls are bounded. A wait that runs out is final for its CTA: it sets Scalars::fault, posts no
// further partial and leaves the launch, so that its teammates' next wait runs out too. What a team
// leaves unsolved keeps Scalars::pending.
// FP64 is slow on this GPU: an FP64 instruction occupies the SM's pipe for 16 clocks a warp and its
// result takes about 100; a division takes about 1000. Measured per iteration of a small body with
// FP64 trees and divisions: 1500 clocks of the update and 1000 of each sum. So sums are integer sums of
// mantissas of 58 bits aligned to the largest (Fixed), rounded to FP64 once at the end, comparisons are
// made on the bits, and alpha and beta of the FP32 modes, which are rounded to float, are divided in
// float-float.
//
// The rows' arithmetic is that of the launches it replaces, in the same order.
#pragma once

#include "device.cuh"
#include "ops.h"

#include <cooperative_groups.h>
#include <type_traits>

namespace b3g {

namespace {

constexpr int kSolveMaxThreads = 512;
constexpr int kL1Room = 32 << 10;             // shared memory left to the L1 where it serves the gathers
constexpr int kPollLimit = 1 << 20;           // polls of L2 before a warp gives up (about a second)
constexpr int kSmemPollLimit = 16 * kPollLimit;  // of its shared memory
constexpr int kTeamWarpSlots = kTeamMax / 32; // slots a lane of the polling warp reads


__device__ __forceinline__ void st_relaxed(unsigned long long p[2], ulonglong2 v)
{
	asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(v.x), "l"(v.y) : "memory");
}
__device__ __forceinline__ ulonglong2 ld_relaxed(const unsigned long long p[2])
{
	ulonglong2 v;
	asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
	return v;
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p)
{
	unsigned v;
	asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
	return v;
}
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void red_release(unsigned* p)
{
	asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}

// m 2^e with |m| < 2^58: a float's or a double's value, or a sum of such values, of each of which 57 bits
// below the largest one's first are kept. Infinities have e >= kNotFinite and m as if they were numbers,
// a NaN's e is kNaN or above and swamps them.
struct Fixed
{
	long long m;
	int e;
};
constexpr int kNotFinite = 1 << 20, kNaN = kNotFinite + 4096, kFixedZero = -(1 << 20);

__device__ __forceinline__ Fixed to_fixed(float t)
{
	const unsigned u = __float_as_uint(t);
	const int e = (int)((u >> 23) & 0xffu);
	const long long m = (long long)((u & 0x7fffffu) | (e > 0 ? 0x800000u : 0u)) << 34;
	Fixed f;
	f.m = (u >> 31) ? -m : m;
	f.e = e == 0xff ? ((u & 0x7fffffu) ? kNaN : kNotFinite) : (m == 0 ? kFixedZero : max(e, 1) - 184);
	return f;
}
__device__ __forceinline__ Fixed to_fixed(double t)
{
	const unsigned long long u = (unsigned long long)__double_as_longlong(t);
	const int e = (int)((u >> 52) & 0x7ffu);
	const long long m = (long long)((u & 0xfffffffffffffull) | (e > 0 ? 0x10000000000000ull : 0ull)) << 5;
	Fixed f;
	f.m = (u >> 63) ? -m : m;
	f.e = e == 0x7ff ? ((u & 0xfffffffffffffull) ? kNaN : kNotFinite) : (m == 0 ? kFixedZero : max(e, 1) - 1080);
	return f;
}
// back below 2^58
__device__ __forceinline__ Fixed fixed_norm(long long m, int e)
{
	const int sh = max(0, 6 - __clzll(m < 0 ? -m : m));
	Fixed f;
	f.m = m >> sh;
	f.e = m == 0 && e < kNotFinite ? kFixedZero : e + sh;
	return f;
}
__device__ __forceinline__ Fixed fixed_add(Fixed a, Fixed b)
{
	const int e = max(a.e, b.e);
	return fixed_norm((a.m >> min(e - a.e, 63)) + (b.m >> min(e - b.e, 63)), e);
}
// the 32 lanes' sum, in all lanes, |m| < 2^63: aligned to the largest exponent, in limbs of 20 bits
// whose sums fit 32 bits
__device__ __forceinline__ Fixed fixed_warp_sum(Fixed a)
{
	Fixed t;
	t.e = __reduce_max_sync(0xffffffffu, a.e);
	const long long q = a.m >> min(t.e - a.e, 63);
	const int l0 = (int)__reduce_add_sync(0xffffffffu, (unsigned)(q & 0xfffff));
	const int l1 = (int)__reduce_add_sync(0xffffffffu, (unsigned)((q >> 20) & 0xfffff));
	const int l2 = __reduce_add_sync(0xffffffffu, (int)(q >> 40));
	t.m = (long long)l0 + ((long long)l1 << 20) + ((long long)l2 << 40);
	return t;
}
// The nearest double (|m| < 2^63): a normal number in a line, what is not one apart
__device__ __noinline__ double fixed_rare(Fixed a)
{
	const unsigned long long u = (unsigned long long)(a.m < 0 ? -a.m : a.m), sign = a.m < 0 ? 1ull << 63 : 0ull;
	if (a.e >= kNotFinite)  // a sum with opposite infinities is what is left of their ms: about 0
		return __longlong_as_double(a.e >= kNaN || u < (1ull << 40) ? 0x7ff8000000000000ll : (long long)(sign | 0x7ff0000000000000ull));
	if (u == 0 || a.e < -1137) return 0.0;
	if (a.e + 63 - __clzll((long long)u) > 1023) return __longlong_as_double((long long)(sign | 0x7ff0000000000000ull));
	// below the normal numbers: a multiple of 2^-1074
	const int drop = -1074 - a.e;
	return __longlong_as_double((long long)(sign | (drop > 0 ? (u + (1ull << (drop - 1))) >> drop : u << -drop)));
}
__device__ __forceinline__ double fixed_value(Fixed a)
{
	const unsigned long long u = (unsigned long long)(a.m < 0 ? -a.m : a.m);
	const int lz = __clzll((long long)u);
	const int ex = a.e - lz + 1085;  // the exponent field less the mantissa's leading bit
	if (u == 0 || (unsigned)ex >= 0x7feu) return fixed_rare(a);
	const unsigned long long r = (((u << lz) >> 10) + 1ull) >> 1;
	return __longlong_as_double((long long)((((unsigned long long)ex << 52) + r) | ((unsigned long long)a.m & (1ull << 63))));
}
// A partial in a slot: mantissa and exponent, each with the sum's two-bit number
__device__ __forceinline__ ulonglong2 fixed_words(Fixed a, unsigned long long tag)
{
	return make_ulonglong2(((unsigned long long)a.m << 2) | tag, ((unsigned long long)(long long)a.e << 2) | tag);
}
__device__ __forceinline__ bool tagged(ulonglong2 w, unsigned long long tag) { return (w.x & 3ull) == tag && (w.y & 3ull) == tag; }
__device__ __forceinline__ Fixed fixed_of(ulonglong2 w)
{
	Fixed a;
	a.m = (long long)w.x >> 2;
	a.e = (int)((long long)w.y >> 2);
	return a;
}

// Comparisons on the bits of doubles (an FP64 comparison waits for the FP64 pipe)
__device__ __forceinline__ bool bits_finite(double x) { return ((__double_as_longlong(x) >> 52) & 0x7ff) != 0x7ff; }
__device__ __forceinline__ bool bits_positive(double x) { return __double_as_longlong(x) > 0; }
// x <= y for finite x and y >= 0
__device__ __forceinline__ bool bits_at_most(double x, double y) { return __double_as_longlong(x) <= __double_as_longlong(y); }

// a / b rounded to the vector type. For float, in double-single arithmetic (Dekker, A floating-point
// technique for extending the available precision, 1971): each mantissa as two floats, the
// denominator's reciprocal as an estimate and its correction. The quotient is good to 2^-42, 2^-18 of
// half a float's unit in the last place; one that close to the midpoint of two floats, or beside a power
// of two, takes the FP64 division (once in about 2^13), so the result is always its result. The
// reciprocal is formed ahead where the denominator is known ahead.
template <class TV>
struct Divisor;
// (a call, so that no part of it is on the way of the others)
__device__ __noinline__ float divide_fp64(double a, double b) { return (float)(a / b); }
template <>
struct Divisor<double>
{
	double b;
	__device__ __forceinline__ explicit Divisor(double v) : b(v) {}
	__device__ __forceinline__ double divide(double a) const { return a / b; }
};
template <>
struct Divisor<float>
{
	double b;
	float hi, lo;
	int e;       // exponent field of b; 0 or 0x7ff: the FP64 division
	bool neg;
	__device__ __forceinline__ explicit Divisor(double v) : b(v)
	{
		const unsigned long long u = (unsigned long long)__double_as_longlong(v);
		e = (int)((u >> 52) & 0x7ff);
		neg = (u >> 63) != 0;
		// mantissa in [1, 2): 23 fraction bits in the high float, 29 in the low one
		const float bh = __uint_as_float(0x3f800000u | (unsigned)((u >> 29) & 0x7fffffu));
		const float bl = (float)(unsigned)(u & 0x1fffffffu) * 0x1p-52f;
		hi = __fdividef(1.0f, bh);
		lo = hi * (fmaf(-bh, hi, 1.0f) - bl * hi);
	}
	__device__ __forceinline__ float divide(double a) const
	{
		const unsigned long long u = (unsigned long long)__double_as_longlong(a);
		const int ea = (int)((u >> 52) & 0x7ff);
		const float ah = __uint_as_float(0x3f800000u | (unsigned)((u >> 29) & 0x7fffffu));
		const float al = (float)(unsigned)(u & 0x1fffffffu) * 0x1p-52f;
		const float q0 = ah * hi;
		const float c = fmaf(ah, hi, -q0) + fmaf(ah, lo, al * hi);
		const float q = q0 + c;
		const unsigned qb = __float_as_uint(q);
		// what the rounding to q left (exact), against half a unit in the last place
		const float left = fabsf((q0 - q) + c), half = __uint_as_float((qb & 0x7f800000u) - (24u << 23));
		const int ex = (int)(qb >> 23) + (ea - e);
		// or a zero, a denormal, a value that is not finite, or a quotient outside the normal floats
		if (left > half * (1.0f - 0x1p-13f) || !(qb & 0x7fffffu) || ea == 0 || ea == 0x7ff || e == 0 || e == 0x7ff || ex <= 0 ||
		    ex >= 0xff)
			return divide_fp64(a, b);
		return __uint_as_float((qb & 0x7fffffu) | ((unsigned)ex << 23) | (((u >> 63) != 0) != neg ? 0x80000000u : 0u));
	}
};

// One row's term of a dot product in the vector type (dot3 widens it)
template <class TV>
__device__ __forceinline__ TV term3(const TV a[3], const TV b[3])
{
	return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

struct SolveSh
{
	Fixed w[2][32];
	double total, ratio;
	int ok, lost;
	int polls;  // of a gather that waits for a version
	ulonglong2 slot[2][kMaxTeamCtas];  // a cluster's partials
	unsigned fenced[kMaxTeamCtas];     // the last sum before which a cluster's CTA has fenced
};

// The sum of a CTA's warps, in warp 0 (v is each warp's value, already in sh->w[buf])
__device__ __forceinline__ Fixed cta_total(const SolveSh* sh, int buf, Fixed v)
{
	const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
	if (nw > 1)
	{
		Fixed z;
		z.m = 0;
		z.e = kFixedZero;
		if (lane < nw) z = sh->w[buf][lane];
		z = fixed_warp_sum(z);
		v = fixed_norm(z.m, z.e);
	}
	return v;
}

// The reduction memory (cleared before the launch) and this CTA's place in the team.
template <class TV>
struct GridTeam
{
	SolveSh* sh;
	TeamMemory* mem;
	int ctas, rank;
	int replicas, polls;
	unsigned sums, fences;  // so far
	int ok;
	TV ratio;

	__device__ __forceinline__ GridTeam(SolveSh* s, TeamMemory* m, int limit)
	    : sh(s), mem(m), ctas(gridDim.x), rank(blockIdx.x), replicas(gridDim.x > 16 ? kTeamReplicas : 1),
	      polls(limit > 0 ? limit : kPollLimit), sums(0), fences(0), ok(1), ratio((TV)0)
	{
		if (threadIdx.x == 0)
		{
			sh->lost = 0;
			sh->polls = polls;
		}
	}

	// This warp's value v (the same in all lanes) summed over the team. `between` runs after this
	// CTA's partial is on its way; ratio_of(total) is evaluated once per CTA and left in `ratio`.
	// FENCE: what the team's threads wrote before the sum may be read by all of them after it.
	template <bool FENCE, class F, class R>
	__device__ __forceinline__ double sum(Fixed v, F between, R ratio_of)
	{
		const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
		const int buf = sums & 1;
		if (lane == 0) sh->w[buf][warp] = v;
		__syncthreads();
		const unsigned long long tag = (unsigned long long)(((sums >> 1) + 1) & 3);
		unsigned long long(*all)[kTeamMax][2] = mem->tagged[buf];
		if (warp == 0)
		{
			const ulonglong2 w = fixed_words(cta_total(sh, buf, v), tag);
			if (lane < replicas) st_relaxed(all[lane][rank], w);
		}
		if (FENCE && threadIdx.x == 0) red_release(&mem->arrived);
		between();
		if (warp == 0)
		{
			unsigned long long(*mine)[2] = all[rank & (replicas - 1)];
			ulonglong2 u[kTeamWarpSlots];
			const ulonglong2 none = fixed_words(Fixed{0, kFixedZero}, tag);
			int tries = 0;
			bool there;
			for (;;)
			{
				there = true;
#pragma unroll
				for (int q = 0; q < kTeamWarpSlots; ++q)
				{
					u[q] = lane + 32 * q < ctas ? ld_relaxed(mine[lane + 32 * q]) : none;
					there = there && tagged(u[q], tag);
				}
				there = __all_sync(0xffffffffu, there) != 0;
				if (there || ++tries > polls) break;
			}
			// a lane's slots aligned to their largest exponent and to 55 bits, so that five of them stay
			// below 2^58
			Fixed f[kTeamWarpSlots], t;
			t.e = kFixedZero;
#pragma unroll
			for (int q = 0; q < kTeamWarpSlots; ++q)
			{
				f[q] = fixed_of(u[q]);
				t.e = max(t.e, f[q].e);
			}
			t.m = 0;
#pragma unroll
			for (int q = 0; q < kTeamWarpSlots; ++q) t.m += (f[q].m >> 3) >> min(t.e - f[q].e, 60);
			t.e += 3;
			const double total = fixed_value(fixed_warp_sum(t));
			const TV r = ratio_of(total);
			if (FENCE)
			{
				const unsigned want = (fences + 1) * (unsigned)ctas;
				while (ld_acquire(&mem->arrived) < want)
					if (++tries > polls)
					{
						there = false;
						break;
					}
				there = __all_sync(0xffffffffu, there) != 0;
			}
			if (lane == 0)
			{
				sh->total = total;
				*(TV*)&sh->ratio = r;
				sh->ok = there && !sh->lost ? 1 : 0;
				if (!there) sh->lost = 1;
			}
		}
		++sums;
		if (FENCE) ++fences;
		__syncthreads();
		ok = sh->ok;
		ratio = *(const TV*)&sh->ratio;
		return sh->total;
	}
	template <bool FENCE>
	__device__ __forceinline__ double sum(Fixed v)
	{
		return sum<FENCE>(v, [] {}, [](double) { return (TV)0; });
	}
	// execution and visibility only
	__device__ __forceinline__ void publish()
	{
		Fixed z;
		z.m = 0;
		z.e = kFixedZero;
		sum<true>(z);
	}
};

// `size` consecutive CTAs of a thread-block cluster from rank `base` (size 1: a CTA by itself).
// Partials go straight into the slots of every member's shared memory, where its warp 0 polls them:
// one trip through the cluster's network a sum. The number's two bits work as in the grid team. A
// team may split into smaller ones between two sums: its members have counted the same sums, and a
// slot's last partial is of the sum two before, so it is told from the next one.
template <class TV>
struct ClusterTeam
{
	SolveSh* sh;
	int cta;          // rank in the cluster
	int rank, base, ctas;
	int polls;
	unsigned sums;
	int ok;
	TV ratio;

	// (the caller synchronises the cluster after this, and again before a CTA leaves the kernel)
	__device__ __forceinline__ ClusterTeam(SolveSh* s, int limit)
	    : sh(s), cta((int)cooperative_groups::this_cluster().block_rank()), rank(0), base(0), ctas(1),
	      polls(limit > 0 ? limit : kSmemPollLimit), sums(0), ok(1), ratio((TV)0)
	{
		if (threadIdx.x < 2 * kMaxTeamCtas) (&sh->slot[0][0])[threadIdx.x] = make_ulonglong2(0ull, 0ull);
		if (threadIdx.x < kMaxTeamCtas) sh->fenced[threadIdx.x] = 0u;
		if (threadIdx.x == 0)
		{
			sh->lost = 0;
			sh->polls = limit > 0 ? limit : kPollLimit;
		}
	}
	// the address of a member's copy of a shared variable
	__device__ __forceinline__ unsigned peer(const void* p, int member) const
	{
		unsigned remote;
		asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
		             : "=r"(remote)
		             : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(base + member));
		return remote;
	}
	__device__ __forceinline__ void form(int size)
	{
		ctas = size;
		base = cta / size * size;
		rank = cta - base;
	}
	template <bool FENCE, class F, class R>
	__device__ __forceinline__ double sum(Fixed v, F between, R ratio_of)
	{
		const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
		const int buf = sums & 1;
		if (lane == 0) sh->w[buf][warp] = v;
		__syncthreads();
		const unsigned long long tag = (unsigned long long)(((sums >> 1) + 1) & 3);
		Fixed t = v;
		if (warp == 0)
		{
			t = cta_total(sh, buf, v);
			if (lane < ctas && ctas > 1)
			{
				const ulonglong2 w = fixed_words(t, tag);
				asm volatile("st.relaxed.cluster.shared::cluster.v2.u64 [%0], {%1, %2};" ::"r"(peer(&sh->slot[buf][rank], lane)), "l"(w.x), "l"(w.y)
				             : "memory");
			}
		}
		if (FENCE && ctas > 1 && threadIdx.x >= blockDim.x - 32)
		{
			fence_gpu();
			if (lane < ctas)
				asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(peer(&sh->fenced[rank], lane)), "r"(sums + 1) : "memory");
		}
		between();
		if (warp == 0)
		{
			bool there = true;
			if (ctas > 1)
			{
				ulonglong2 u = fixed_words(Fixed{0, kFixedZero}, tag);
				unsigned fenced = sums + 1;
				const unsigned mine = (unsigned)__cvta_generic_to_shared(&sh->slot[buf][lane < ctas ? lane : 0]);
				const unsigned flag = (unsigned)__cvta_generic_to_shared(&sh->fenced[lane < ctas ? lane : 0]);
				for (int tries = 0;;)
				{
					if (lane < ctas)
					{
						asm volatile("ld.relaxed.cluster.shared::cta.v2.u64 {%0, %1}, [%2];" : "=l"(u.x), "=l"(u.y) : "r"(mine) : "memory");
						if (FENCE) asm volatile("ld.relaxed.cluster.shared::cta.u32 %0, [%1];" : "=r"(fenced) : "r"(flag) : "memory");
					}
					there = __all_sync(0xffffffffu, tagged(u, tag) && (int)(fenced - (sums + 1)) >= 0) != 0;
					if (there || ++tries > polls) break;
				}
				t = fixed_warp_sum(fixed_of(u));
				if (FENCE) fence_gpu();
			}
			const double total = fixed_value(t);
			const TV r = ratio_of(total);
			if (lane == 0)
			{
				sh->total = total;
				*(TV*)&sh->ratio = r;
				sh->ok = there && !sh->lost ? 1 : 0;
				if (!there) sh->lost = 1;
			}
		}
		++sums;
		__syncthreads();
		ok = sh->ok;
		ratio = *(const TV*)&sh->ratio;
		return sh->total;
	}
	template <bool FENCE>
	__device__ __forceinline__ double sum(Fixed v)
	{
		return sum<FENCE>(v, [] {}, [](double) { return (TV)0; });
	}
	__device__ __forceinline__ void publish()
	{
		Fixed z;
		z.m = 0;
		z.e = kFixedZero;
		sum<true>(z);
	}
	// the first member's thread 0 evaluates next() (an integer below 2^30), the team returns it
	template <class N>
	__device__ __forceinline__ int agree(N next)
	{
		Fixed z;
		z.m = 0;
		z.e = kFixedZero;
		if (rank == 0 && threadIdx.x < 32)
		{
			int item = threadIdx.x == 0 ? next() : 0;
			item = __shfl_sync(0xffffffffu, item, 0);
			z.m = (long long)item << 20;
			z.e = item ? -20 : kFixedZero;
		}
		return (int)sum<false>(z);
	}
};

// A vertex's s with the number of its version in the fourth component, as one 16-byte access each
// way: the versions of a vector are told apart without a barrier.
__device__ __forceinline__ float4 ld_version(const float* s, int i)
{
	unsigned long long lo, hi;
	asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
	             : "=l"(lo), "=l"(hi)
	             : "l"(s + 4 * (size_t)i)
	             : "memory");
	return make_float4(__uint_as_float((unsigned)lo), __uint_as_float((unsigned)(lo >> 32)), __uint_as_float((unsigned)hi),
	                   __uint_as_float((unsigned)(hi >> 32)));
}
__device__ __forceinline__ void st_version(float* s, int i, const float o[3], unsigned version)
{
	const unsigned long long lo = (unsigned long long)__float_as_uint(o[0]) | ((unsigned long long)__float_as_uint(o[1]) << 32);
	const unsigned long long hi = (unsigned long long)__float_as_uint(o[2]) | ((unsigned long long)version << 32);
	asm volatile("{ .reg .b128 t; mov.b128 t, {%0, %1}; st.relaxed.gpu.global.b128 [%2], t; }" ::"l"(lo), "l"(hi),
	             "l"(s + 4 * (size_t)i)
	             : "memory");
}

// How a sweep gathers s (team_spmv_row): by its versions, or with the loads of a policy from a vector
// that a fenced sum has published.
struct GatherVersions
{
};
// A sweep whose matrix comes from L2 shares the L2-to-SM network with its gathers, a fourth of its
// bytes, and a vertex is gathered about 15 times, mostly by one SM: with many warps (DEPTH 1) the FP32
// sweep gathers through the L1, and the launch leaves it kL1Room of the SM's memory. Other SMs write what
// it reads, so each new s is fenced. ms a step by versions from L2 / by versions through the L1, which is a
// race (the loads' scope is not the stores') / behind fences: 64^3 block 9.6 / 9.4 / 9.3, BF16 block of
// 47x41x37 3.55 / 3.40 / 3.26, 160 blocks 10.3 / 10.0 / 10.1, 16 blocks and cloths 5.87 / 5.58 / 5.61, 12
// blocks 1.42 / 1.38 / 1.44.
template <class TV, int DEPTH>
struct GatherOf
{
	typedef typename std::conditional<sizeof(TV) == 8, LdCG, typename std::conditional<DEPTH == 1, LdPlain, GatherVersions>::type>::type type;
};

// Where a slice's matrix comes from: shared memory (a chunk of nine planes and the column ids of
// its w x 32 slots) or global memory with an L2 policy.
template <class TA>
struct SmemMat
{
	const unsigned char* chunk;
	int slots;
	__device__ __forceinline__ int4 cols(int off) const { return *(const int4*)(chunk + (size_t)9 * slots * sizeof(TA) + 4 * (size_t)off); }
	__device__ __forceinline__ void plane(int p, int off, typename Acc<TA>::type o[4]) const
	{
		load4<TA, LdPlain>((const TA*)chunk + (size_t)p * slots + off, o);
	}
};
template <class TA>
struct GlobalMat
{
	const TA* A;
	const int* col;
	size_t ns;
	size_t base;
	unsigned long long pol;
	__device__ __forceinline__ int4 cols(int off) const { return hinted_cols<MatNC>(col + base + off, pol); }
	__device__ __forceinline__ void plane(int p, int off, typename Acc<TA>::type o[4]) const
	{
		hinted_load4<MatNC>(A + p * ns + base + off, o, pol);
	}
};

// o = (A s)_i and own = s_i (the diagonal block leads every row); the products are summed in slot
// order, as spmv_row sums them. G: how s is gathered; of a vector with versions, entries older than
// `version` are read again (sh->lost: a wait ran out).
// DEPTH groups of four blocks have their columns' s in flight at a time: the gathers go to L2, and a
// thread that waits for them group by group pays that trip four times a row (matrix in shared
// memory, few warps). With DEPTH 1 (many warps, matrix from L2) the column ids are read a group
// ahead, so that a group's planes and gathers are in flight together.
template <class TA, class TV, int DEPTH, class G, class M>
__device__ __forceinline__ void team_spmv_row(const M& m, int w, int lane, const TV* s, unsigned version, SolveSh* sh,
                                              TV o[3], TV own[3])
{
	typedef typename Acc<TA>::type AT;
	AT o0 = 0, o1 = 0, o2 = 0;
	int4 ahead;
	if (DEPTH == 1) ahead = m.cols(4 * lane);
	for (int k0 = 0; k0 < w; k0 += DEPTH * kGroup)
	{
		AT a[9][4];
		int jj[DEPTH][4];
		if (DEPTH == 1)
		{
#pragma unroll
			for (int p = 0; p < 9; ++p) m.plane(p, 32 * k0 + 4 * lane, a[p]);
		}
#pragma unroll
		for (int g = 0; g < DEPTH; ++g)
			if (g == 0 || k0 + g * kGroup < w)
			{
				const int4 c = DEPTH == 1 ? ahead : m.cols(32 * (k0 + g * kGroup) + 4 * lane);
				jj[g][0] = c.x;
				jj[g][1] = c.y;
				jj[g][2] = c.z;
				jj[g][3] = c.w;
			}
		TV xv[DEPTH][4][3];
		if constexpr (std::is_same<G, GatherVersions>::value)
		{
			float4 r[DEPTH][4];
#pragma unroll
			for (int g = 0; g < DEPTH; ++g)
				if (g == 0 || k0 + g * kGroup < w)
#pragma unroll
					for (int u = 0; u < 4; ++u) r[g][u] = ld_version(s, jj[g][u]);
			for (int polls = 0;; ++polls)
			{
				bool old = false;
#pragma unroll
				for (int g = 0; g < DEPTH; ++g)
					if (g == 0 || k0 + g * kGroup < w)
#pragma unroll
						for (int u = 0; u < 4; ++u)
							if (__float_as_uint(r[g][u].w) != version)
							{
								r[g][u] = ld_version(s, jj[g][u]);
								old = true;
							}
				if (!old) break;
				if (polls > sh->polls || *(volatile int*)&sh->lost)
				{
					sh->lost = 1;
					break;
				}
			}
#pragma unroll
			for (int g = 0; g < DEPTH; ++g)
#pragma unroll
				for (int u = 0; u < 4; ++u)
				{
					xv[g][u][0] = r[g][u].x;
					xv[g][u][1] = r[g][u].y;
					xv[g][u][2] = r[g][u].z;
				}
		}
		else
		{
#pragma unroll
			for (int g = 0; g < DEPTH; ++g)
				if (g == 0 || k0 + g * kGroup < w)
#pragma unroll
					for (int u = 0; u < 4; ++u) vld<TV, G>(s, jj[g][u], xv[g][u]);
			if (DEPTH == 1 && k0 + kGroup < w) ahead = m.cols(32 * (k0 + kGroup) + 4 * lane);
		}
		if (k0 == 0)
		{
#pragma unroll
			for (int c = 0; c < 3; ++c) own[c] = xv[0][0][c];
		}
#pragma unroll
		for (int g = 0; g < DEPTH; ++g)
			if (g == 0 || k0 + g * kGroup < w)
			{
				if (DEPTH > 1)
				{
#pragma unroll
					for (int p = 0; p < 9; ++p) m.plane(p, 32 * (k0 + g * kGroup) + 4 * lane, a[p]);
				}
#pragma unroll
				for (int u = 0; u < 4; ++u)
				{
					const AT x0 = (AT)xv[g][u][0], x1 = (AT)xv[g][u][1], x2 = (AT)xv[g][u][2];
					o0 += a[0][u] * x0 + a[1][u] * x1 + a[2][u] * x2;
					o1 += a[3][u] * x0 + a[4][u] * x1 + a[5][u] * x2;
					o2 += a[6][u] * x0 + a[7][u] * x1 + a[8][u] * x2;
				}
			}
	}
	o[0] = (TV)o0;
	o[1] = (TV)o1;
	o[2] = (TV)o2;
}

// (A x)_i in float-float from the float-float x (spmv_row_ff), x read through L2
template <class M>
__device__ __forceinline__ void team_spmv_row_ff(const M& m, int w, int lane, const float* xff, float ohi[3], float olo[3])
{
	float h0 = 0, h1 = 0, h2 = 0, l0 = 0, l1 = 0, l2 = 0;
	for (int k = 0; k < w; k += kGroup)
	{
		const int off = 32 * k + 4 * lane;
		const int4 jj = m.cols(off);
		float a[9][4];
#pragma unroll
		for (int p = 0; p < 9; ++p) m.plane(p, off, a[p]);
		const int js[4] = {jj.x, jj.y, jj.z, jj.w};
#pragma unroll
		for (int u = 0; u < 4; ++u)
		{
			float xh[3], xl[3];
			vld<float, LdCG>(xff, 2 * js[u], xh);
			vld<float, LdCG>(xff, 2 * js[u] + 1, xl);
#pragma unroll
			for (int c = 0; c < 3; ++c)
			{
				const float a0 = a[3 * 0 + c][u], a1 = a[3 * 1 + c][u], a2 = a[3 * 2 + c][u];
				float p = __fmul_rn(a0, xh[c]);
				ff_add(h0, l0, p, fmaf(a0, xh[c], -p) + a0 * xl[c]);
				p = __fmul_rn(a1, xh[c]);
				ff_add(h1, l1, p, fmaf(a1, xh[c], -p) + a1 * xl[c]);
				p = __fmul_rn(a2, xh[c]);
				ff_add(h2, l2, p, fmaf(a2, xh[c], -p) + a2 * xl[c]);
			}
		}
	}
	ohi[0] = h0; ohi[1] = h1; ohi[2] = h2;
	olo[0] = l0; olo[1] = l1; olo[2] = l2;
}

// Bytes of shared memory per slot of the matrix, and per slice of the row-local vectors: r, d, q
// and the scalar Jacobi (4-wide), x (4-wide, or 8 floats in float-float).
template <class TA>
__host__ __device__ constexpr int solve_slot_bytes() { return 9 * (int)sizeof(TA) + 4; }
template <class TV, bool FF>
__host__ __device__ constexpr int solve_vec_bytes() { return 32 * (4 * 4 + (FF ? 8 : 4)) * (int)sizeof(TV); }
// the BF16 mode's: r, q, p, the Jacobi and x of the outer iteration, r, d, q and z of the inner one
constexpr int kFcgVecBytes = 32 * (8 * 4 + 8) * (int)sizeof(float);

// One lane's row vectors in shared memory or in the body's arrays.
template <class TV, bool FF>
struct RowVecs
{
	TV *r, *d, *q, *m, *x;
	__device__ __forceinline__ RowVecs(const DevBody& B, unsigned char* vec, int j, int vec_slices, int lane, int i)
	{
		if (j < vec_slices)
		{
			TV* p = (TV*)(vec + (size_t)j * solve_vec_bytes<TV, FF>());
			r = p + 4 * lane;
			d = p + 128 + 4 * lane;
			q = p + 256 + 4 * lane;
			m = p + 384 + 4 * lane;
			x = p + 512 + (FF ? 8 : 4) * lane;
		}
		else
		{
			r = (TV*)B.r + 4 * (size_t)i;
			d = (TV*)B.d + 4 * (size_t)i;
			q = (TV*)B.q + 4 * (size_t)i;
			m = (TV*)B.Minv + 4 * (size_t)i;
			x = FF ? (TV*)B.xff + 8 * (size_t)i : (TV*)B.py + 4 * (size_t)i;
		}
	}
};

struct FcgRowVecs
{
	float *r, *q, *p, *m, *x, *ri, *di, *qi, *z;
	__device__ __forceinline__ FcgRowVecs(const DevBody& B, const FcgVecs& W, unsigned char* vec, int j, int vec_slices,
	                                      int lane, int i)
	{
		if (j < vec_slices)
		{
			float* b = (float*)(vec + (size_t)j * kFcgVecBytes) + 4 * lane;
			r = b;
			q = b + 128;
			p = b + 256;
			m = b + 384;
			ri = b + 512;
			di = b + 640;
			qi = b + 768;
			z = b + 896;
			x = b + 1024 + 4 * lane;
		}
		else
		{
			const size_t o = 4 * (size_t)i;
			r = (float*)B.r + o;
			q = (float*)B.q + o;
			p = (float*)B.d + o;
			m = (float*)B.Minv + o;
			ri = W.r + o;
			di = W.d + o;
			qi = W.q + o;
			z = W.z + o;
			x = B.xff + 2 * o;
		}
	}
};

// The slices a CTA owns, which of them keep their vectors and their matrix (of storage type TA)
// in shared memory: vectors first, since every iteration reads and writes them, then matrices.
template <class TA>
struct OwnSlices
{
	const DevBody& B;
	const TA* A;
	int s0, ns, base0, vec_slices, mat_slices;
	unsigned char *vec, *mat;
	unsigned long long pol, keep_pol;
	int keep_slices;  // local slices below it are kept in L2 (keep_pol), the others stream through it

	__device__ __forceinline__ OwnSlices(const DevBody& body, const TA* a, unsigned char* smem, int room, int vecb, int keep,
	                                     int rank, int ctas)
	    : B(body), A(a)
	{
		s0 = (int)((long long)rank * B.nslices / ctas);
		ns = (int)((long long)(rank + 1) * B.nslices / ctas) - s0;
		vec_slices = min(ns, room / vecb);
		vec = smem;
		mat = smem + (size_t)vec_slices * vecb;
		base0 = B.slice_ptr[s0];
		mat_slices = 0;
		pol = evict_first_policy();
		keep_pol = keep < 1024 ? evict_last_policy() : evict_normal_policy();
		keep_slices = (int)((long long)ns * keep >> 10);
		if (vec_slices < ns) return;
		const int cap = (room - vec_slices * vecb) / solve_slot_bytes<TA>();
		int lo = 0, hi = ns;
		while (lo < hi)
		{
			const int mid = (lo + hi + 1) >> 1;
			if (B.slice_ptr[s0 + mid] - base0 <= cap) lo = mid;
			else hi = mid - 1;
		}
		mat_slices = lo;
	}
	// the cached matrices, each copied by the warp that will read it
	__device__ __forceinline__ void load() const
	{
		const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
		for (int j = threadIdx.x >> 5; j < mat_slices; j += nw)
		{
			const int base = B.slice_ptr[s0 + j], slots = B.slice_ptr[s0 + j + 1] - base;
			unsigned char* c = mat + (size_t)(base - base0) * solve_slot_bytes<TA>();
			constexpr int kPer = 16 / (int)sizeof(TA);
			for (int p = 0; p < 9; ++p)
				for (int k = lane; k < slots / kPer; k += 32)
					((uint4*)c)[(size_t)p * (slots / kPer) + k] = mat_ld16<MatNC>(A + (size_t)p * B.nslots + base + k * kPer, pol);
			uint4* cc = (uint4*)(c + (size_t)9 * slots * sizeof(TA));
			for (int k = lane; k < slots / 4; k += 32) cc[k] = mat_ld16<MatNC>(B.col + base + 4 * k, pol);
		}
		__syncwarp();
	}
	// f(local slice j, row i) for the rows of this warp's slices
	template <class F>
	__device__ __forceinline__ void rows(F f) const
	{
		const int nw = blockDim.x >> 5;
		for (int j = threadIdx.x >> 5; j < ns; j += nw)
		{
			const int i = (s0 + j) * kSlice + (threadIdx.x & 31);
			if (i < B.n) f(j, i);
		}
	}
	// the sum of f(j, i), a term of type T per row, over this warp's rows; all lanes return it
	template <class T, class F>
	__device__ __forceinline__ Fixed row_sum(F f) const
	{
		const int nw = blockDim.x >> 5;
		Fixed s;
		s.m = 0;
		s.e = kFixedZero;
		for (int j = threadIdx.x >> 5; j < ns; j += nw)
		{
			const int i = (s0 + j) * kSlice + (threadIdx.x & 31);
			T t = (T)0;
			if (i < B.n) t = f(j, i);
			const Fixed w = fixed_warp_sum(to_fixed(t));
			s = fixed_add(s, fixed_norm(w.m, w.e));
		}
		return s;
	}
	// f(matrix of local slice j, its width)
	template <class F>
	__device__ __forceinline__ void matrix(int j, F f) const
	{
		const int base = B.slice_ptr[s0 + j];
		const int slots = B.slice_ptr[s0 + j + 1] - base;
		if (j < mat_slices) f(SmemMat<TA>{mat + (size_t)(base - base0) * solve_slot_bytes<TA>(), slots}, slots / kSlice);
		else f(GlobalMat<TA>{A, B.col, (size_t)B.nslots, (size_t)base, j < keep_slices ? keep_pol : pol}, slots / kSlice);
	}
};

template <class TV>
__device__ __forceinline__ void row_precond(const DevBody& B, const TV* m, int i, const TV r[3], TV s[3])
{
	if (B.precond == B3G_PRECOND_BLOCK_JACOBI)
	{
		precond_row<TV>(B, i, r, s);
		return;
	}
	TV mm[3];
	vld<TV, LdPlain>(m, 0, mm);
#pragma unroll
	for (int c = 0; c < 3; ++c) s[c] = mm[c] * r[c];
}

template <class TV, bool FF>
__device__ __forceinline__ void row_x_update(TV* x, const TV* dp, TV alpha)
{
	TV d[3];
	vld<TV, LdPlain>(dp, 0, d);
	if constexpr (FF)
	{
		// refinement: the solution accumulates in float-float (the product alpha d and its
		// rounding error are both added)
		float xh[3], xl[3];
		ff_ld(x, 0, xh, xl);
#pragma unroll
		for (int c = 0; c < 3; ++c)
		{
			const float p = __fmul_rn(alpha, d[c]);
			ff_add(xh[c], xl[c], p, fmaf(alpha, d[c], -p));
		}
		ff_st(x, 0, xh, xl);
	}
	else
	{
		TV xx[3];
		vld<TV, LdPlain>(x, 0, xx);
#pragma unroll
		for (int c = 0; c < 3; ++c) xx[c] += alpha * d[c];
		vst(x, 0, xx);
	}
}

// The row's solution as the velocity change dv
template <class TV, bool FF>
__device__ __forceinline__ float3 row_dv(const TV* x)
{
	if constexpr (FF)
	{
		float yh[3], yl[3];
		ff_ld(x, 0, yh, yl);
		return f3(yh[0] + yl[0], yh[1] + yl[1], yh[2] + yl[2]);
	}
	else
	{
		TV y[3];
		vld<TV, LdPlain>(x, 0, y);
		return f3((float)y[0], (float)y[1], (float)y[2]);
	}
}

struct SolveEnd
{
	int status, iter;
	double delta, delta0;
};

// What follows a solve: in a body step the final update (sparse_force_solver.cpp:194-223), which
// with a single Newton iteration also ends the step, or else the Newton loop's exit test and, when
// it ends, the step's end; then the statistics. rows(f) calls f(row i, dv) for this warp's rows,
// update(i, dv, whether the step ends) is the final update of a row.
template <class G, class R, class V>
__device__ __forceinline__ void team_end(G& T, const DevBody& B, const SolveArgs& P, const SolveEnd& S, R rows, V update)
{
	Scalars* sc = B.sc;
	const bool lead = T.rank == 0 && threadIdx.x == 0;
	if (P.newton >= 0)
	{
		bool finish = P.newton_max == 1;
		double part = 0.0;
		rows([&](int i, float3 dv) { part += update(i, dv, finish); });
		const Fixed ws = fixed_warp_sum(to_fixed(part));
		const double err = T.template sum<false>(fixed_norm(ws.m, ws.e));
		const double err0 = P.newton == 0 ? err : sc->newton_err0;
		const bool ndone = P.newton == 0 ? err <= P.newton_tol2 : err <= P.newton_tol2 * err0;
		if (!finish && (ndone || !P.forces_left))
		{
			finish = true;
			rows([&](int i, float3) { post_vertex<LdPlain>(B, i, P.h); });
		}
		if (lead)
		{
			sc->newton_err = err;
			sc->newton_err0 = err0;
			sc->min_it = P.newton == 0 ? S.iter : min(sc->min_it, S.iter);
			sc->max_it = P.newton == 0 ? S.iter : max(sc->max_it, S.iter);
			sc->newton_iter = P.newton + 1;
			sc->total_iters += (unsigned long long)S.iter;
			if (finish) sc->total_steps += 1ull;
			sc->newton_done = finish ? 1 : 0;
		}
	}
	if (lead)
	{
		sc->iter = S.iter;
		sc->delta = S.delta;
		sc->delta0 = S.delta0;
		sc->status = S.status;
		sc->pending = 0;
	}
	if (!T.ok && threadIdx.x == 0) sc->fault = 1;
}

// A sum that never completed: the step's results are not valid (DEVICE_TIMEOUT)
__device__ __forceinline__ void team_fault(const DevBody& B)
{
	B.sc->fault = 1;
	B.sc->newton_done = 1;
}

// sparse_solver.cpp:57-73: whether a solve is over before its first iteration
__device__ __forceinline__ bool solve_over(double delta0, double tol2, int max_iter, int& status)
{
	status = B3G_SOLVE_CONVERGED;
	if (!isfinite(delta0)) status = B3G_SOLVE_NONFINITE;
	else if (delta0 <= tol2 * delta0) status = B3G_SOLVE_CONVERGED;
	else if (max_iter <= 0) status = B3G_SOLVE_MAX_ITERATIONS;
	else return false;
	return true;
}

// Phases timed by the optional instrumentation of the batch kernels (cycles of thread 0 of each CTA,
// barriers and reductions included in the phase that ends with them). The direction update runs
// inside the SpMV sweep, so kPhDir stays zero; its slot keeps the numbering the host reads.
enum { kPhElem = 0, kPhAsm = 1, kPhSpmv = 2, kPhUpdate = 3, kPhDir = 4, kPhFinal = 5, kPhIdle = 6, kPhases = 8 };

// The PCG of one body by one team (sparse_solver.cpp:57-108) and what follows it. update: team_end;
// tick(phase): the phase's end.
template <class TA, class TV, bool FF, int DEPTH, class Team, class V, class C>
__device__ __forceinline__ void team_solve(Team& T, const DevBody& B, const SolveArgs& P, unsigned char* smem, V update, C tick)
{
	typedef RowVecs<TV, FF> Row;
	const int lane = threadIdx.x & 31;
	const OwnSlices<TA> O(B, sizeof(TA) == sizeof(float) ? (const TA*)B.A32 : (const TA*)B.Alo, smem, P.smem,
	                      solve_vec_bytes<TV, FF>(), P.keep, T.rank, T.ctas);
	const TV* sv = (const TV*)B.s;
	// s carries its version, 0 as the assembly leaves it, or every new s is fenced
	typedef typename GatherOf<TV, DEPTH>::type Gather;
	constexpr bool kVersions = std::is_same<Gather, GatherVersions>::value;
	constexpr bool kFence = !kVersions;
	// BF16 blocks: the refresh uses the FP32 ones, and a residual that met the tolerance is confirmed
	// by a refresh before the solve ends
	constexpr bool kConfirm = sizeof(TA) == 2;
	bool confirm = false;
	unsigned version = 0;
	auto store_s = [&](int i, const TV* o) {
		if constexpr (kVersions) st_version((float*)B.s, i, o, version);
		else vst((TV*)B.s, i, o);
	};
	auto row = [&](int j, int i) { return Row(B, O.vec, j, O.vec_slices, lane, i); };

	auto refresh_matrix = [&](int j, auto f) {
		if constexpr (kConfirm)
		{
			const int base = B.slice_ptr[O.s0 + j];
			f(GlobalMat<float>{B.A32, B.col, (size_t)B.nslots, (size_t)base, O.pol}, (B.slice_ptr[O.s0 + j + 1] - base) / kSlice);
		}
		else
			O.matrix(j, f);
	};
	// r = b - A x and s = M^-1 r with x in global memory; this warp's part of r.s
	auto residual = [&]() -> Fixed {
		return O.template row_sum<TV>([&](int j, int i) {
			const Row v = row(j, i);
			TV b[3], rr[3], ss[3];
			vld<TV, LdPlain>((const TV*)B.pb, i, b);
			refresh_matrix(j, [&](const auto& m, int w) {
				if constexpr (FF)
				{
					float qh[3], ql[3];
					team_spmv_row_ff(m, w, lane, B.xff, qh, ql);
#pragma unroll
					for (int c = 0; c < 3; ++c) rr[c] = ff_residual(b[c], qh[c], ql[c]);
				}
				else
				{
					TV q[3], own[3];
					team_spmv_row<typename std::conditional<kConfirm, float, TA>::type, TV, 1, LdCG>(m, w, lane, (const TV*)B.py, 0u, T.sh, q, own);
#pragma unroll
					for (int c = 0; c < 3; ++c) rr[c] = b[c] - q[c];
				}
			});
			row_precond<TV>(B, v.m, i, rr, ss);
			vst(v.r, 0, rr);
			store_s(i, ss);
			return term3(rr, ss);
		});
	};
	// the rows' x to global memory, where a refresh gathers it
	auto publish_x = [&] {
		O.rows([&](int j, int i) {
			if (j >= O.vec_slices) return;
			const Row v = row(j, i);
			if constexpr (FF)
			{
				float xh[3], xl[3];
				ff_ld(v.x, 0, xh, xl);
				ff_st(B.xff, i, xh, xl);
			}
			else
			{
				TV x[3];
				vld<TV, LdPlain>(v.x, 0, x);
				vst((TV*)B.py, i, x);
			}
		});
	};
	auto update_x = [&](TV alpha) {
		O.rows([&](int j, int i) {
			const Row v = row(j, i);
			row_x_update<TV, FF>(v.x, v.d, alpha);
		});
	};

	O.load();
	// the rows' vectors: the assembly left s = M^-1 b for a start from x = 0 (r = b); a warm start
	// takes x as it is
	Fixed part = O.template row_sum<TV>([&](int j, int i) {
		const Row v = row(j, i);
		TV t[3];
		if (j < O.vec_slices && B.precond != B3G_PRECOND_BLOCK_JACOBI)
		{
			vld<TV, LdPlain>((const TV*)B.Minv, i, t);
			vst(v.m, 0, t);
		}
		if (P.warm)
		{
			if (j >= O.vec_slices) return (TV)0;
			if constexpr (FF)
			{
				float xh[3], xl[3];
				ff_ld(B.xff, i, xh, xl);
				ff_st(v.x, 0, xh, xl);
			}
			else
			{
				vld<TV, LdPlain>((const TV*)B.py, i, t);
				vst(v.x, 0, t);
			}
			return (TV)0;
		}
		const TV zero[3] = {0, 0, 0};
		TV ss[3];
		vld<TV, LdPlain>((const TV*)B.pb, i, t);
		vst(v.r, 0, t);
		vld<TV, LdPlain>(sv, i, ss);
		if constexpr (FF) ff_st(v.x, 0, zero, zero);
		else vst(v.x, 0, zero);
		return term3(t, ss);
	});
	if (P.warm)
	{
		// the earlier s may carry any version: fenced once
		++version;
		part = residual();
		T.publish();
	}
	SolveEnd S;
	S.iter = 0;
	S.delta = S.delta0 = T.template sum<false>(part);
	bool done = solve_over(S.delta0, P.tol2, P.max_iter, S.status);
	const double enough = P.tol2 * S.delta0;
	TV beta = (TV)0;
	while (!done && T.ok)
	{
		const bool first = S.iter == 0;
		part = O.template row_sum<TV>([&](int j, int i) {
			const Row v = row(j, i);
			TV o[3], dn[3];
			O.matrix(j, [&](const auto& m, int w) { team_spmv_row<TA, TV, DEPTH, Gather>(m, w, lane, sv, version, T.sh, o, dn); });
			if (!first)
			{
				TV dp[3], qp[3];
				vld<TV, LdPlain>(v.d, 0, dp);
				vld<TV, LdPlain>(v.q, 0, qp);
#pragma unroll
				for (int c = 0; c < 3; ++c)
				{
					dn[c] = dn[c] + beta * dp[c];
					o[c] = o[c] + beta * qp[c];
				}
			}
			vst(v.q, 0, o);
			vst(v.d, 0, dn);
			return term3(dn, o);
		});
		const double dq = T.template sum<false>(part, [] {}, [&](double t) { return Divisor<TV>(t).divide(S.delta); });
		tick(kPhSpmv);
		if (!T.ok) break;
		if (!bits_finite(dq))
		{
			S.status = B3G_SOLVE_NONFINITE;
			break;
		}
		if (!bits_positive(dq))
		{
			S.status = B3G_SOLVE_BREAKDOWN;
			break;
		}
		const TV alpha = T.ratio;
		const Divisor<TV> by_delta(S.delta);
		auto beta_of = [&](double t) { return by_delta.divide(t); };
		double dn;
		const bool refresh = (P.refresh > 0 && (S.iter % P.refresh) == 0) || (kConfirm && confirm);
		if (refresh)
		{
			// sparse_solver.cpp:83-90: r = b - A x
			update_x(alpha);
			publish_x();
			T.publish();
			if (!T.ok) break;
			++version;
			part = residual();
			dn = T.template sum<kFence>(part, [] {}, beta_of);
		}
		else
		{
			++version;
			part = O.template row_sum<TV>([&](int j, int i) {
				const Row v = row(j, i);
				TV r[3], q[3], s[3];
				vld<TV, LdPlain>(v.r, 0, r);
				vld<TV, LdPlain>(v.q, 0, q);
#pragma unroll
				for (int c = 0; c < 3; ++c) r[c] -= alpha * q[c];
				row_precond<TV>(B, v.m, i, r, s);
				vst(v.r, 0, r);
				store_s(i, s);
				return term3(r, s);
			});
			dn = T.template sum<kFence>(part, [&] { update_x(alpha); }, beta_of);
		}
		tick(kPhUpdate);
		beta = T.ratio;
		S.delta = dn;
		S.iter += 1;
		if (!bits_finite(dn)) S.status = B3G_SOLVE_NONFINITE;
		else if (bits_at_most(dn, enough) && (!kConfirm || refresh)) S.status = B3G_SOLVE_CONVERGED;
		else if (S.iter >= P.max_iter) S.status = B3G_SOLVE_MAX_ITERATIONS;
		else
		{
			if (kConfirm) confirm = bits_at_most(dn, enough);
			continue;
		}
		break;
	}
	if (!T.ok)
	{
		team_fault(B);
		return;
	}
	if (P.newton < 0 || P.forces_left) publish_x();  // the result, or the next iteration's start
	team_end(T, B, P, S, [&](auto f) {
		O.rows([&](int j, int i) { f(i, row_dv<TV, FF>(row(j, i).x)); });
	}, update);
	tick(kPhFinal);
}


template <class TA, class TV, bool FF, bool FILTER, int THREADS>
__global__ void __launch_bounds__(THREADS, 1) k_solve(DevBody B, SolveArgs P)
{
	extern __shared__ __align__(16) unsigned char smem[];
	__shared__ SolveSh sh;
	if (P.newton > 0 && B.sc->newton_done) return;
	constexpr int kDepth = THREADS <= 256 ? (sizeof(TV) == 8 ? 2 : 4) : 1;
	GridTeam<TV> T(&sh, B.team, P.polls);
	team_solve<TA, TV, FF, kDepth>(
	    T, B, P, smem,
	    [&](int i, float3 dv, bool finish) { return final_vertex_dv<LdPlain, FILTER>(B, i, P.h, P.newton == 0, finish, dv); },
	    [](int) {});
}

// The same by one cluster, for a body whose slices fit a few CTAs: sums through distributed shared
// memory instead of L2.
template <class TA, class TV, bool FF, bool FILTER>
__global__ void __launch_bounds__(256, 1) k_solve_cluster(DevBody B, SolveArgs P)
{
	extern __shared__ __align__(16) unsigned char smem[];
	__shared__ SolveSh sh;
	ClusterTeam<TV> T(&sh, P.polls);
	cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
	cl.sync();
	if (P.newton <= 0 || !B.sc->newton_done)
	{
		T.form((int)cl.num_blocks());
		team_solve<TA, TV, FF, sizeof(TV) == 8 ? 2 : 4>(
		    T, B, P, smem,
		    [&](int i, float3 dv, bool finish) { return final_vertex_dv<LdPlain, FILTER>(B, i, P.h, P.newton == 0, finish, dv); },
		    [](int) {});
	}
	cl.sync();
}

// The BF16 mode's solve: a flexible CG (Notay's, one stored direction) on the FP32 blocks, with
// float-float x, preconditioned by a fixed number of Jacobi-PCG iterations with the BF16 blocks
// from z = 0. Per outer iteration: z = P(r), p = z - (z.q_prev / p_prev.q_prev) p_prev, q = A p,
// alpha = p.r / p.q, x += alpha p, r -= alpha q or, when a refresh is due, r = b - A x. The BF16
// blocks, read most often, are what is kept in shared memory; the FP32 blocks stream. With 256 threads
// (255 registers) it spills 196 bytes.
template <bool FILTER, int THREADS>
__global__ void __launch_bounds__(THREADS, 1) k_solve_fcg(DevBody B, FcgVecs W, SolveArgs P, int inner)
{
	extern __shared__ __align__(16) unsigned char smem[];
	__shared__ SolveSh sh;
	if (P.newton > 0 && B.sc->newton_done) return;
	typedef FcgRowVecs Row;
	constexpr int kDepth = THREADS <= 256 ? 4 : 1;
	typedef typename GatherOf<float, kDepth>::type Gather;
	constexpr bool kVersions = std::is_same<Gather, GatherVersions>::value;
	typedef __nv_bfloat16 TA;
	const int lane = threadIdx.x & 31;
	GridTeam<float> T(&sh, B.team, P.polls);
	const OwnSlices<TA> O(B, (const TA*)B.Alo, smem, P.smem, kFcgVecBytes, P.keep, T.rank, T.ctas);
	const float* sv = (const float*)B.s;
	unsigned version = 0;  // of s
	const float* pv = (const float*)B.d2;
	auto store_s = [&](int i, const float* o) {
		if constexpr (kVersions) st_version((float*)B.s, i, o, version);
		else vst((float*)B.s, i, o);
	};
	auto row = [&](int j, int i) { return Row(B, W, O.vec, j, O.vec_slices, lane, i); };
	auto matrix32 = [&](int j, auto f) {
		const int base = B.slice_ptr[O.s0 + j];
		f(GlobalMat<float>{B.A32, B.col, (size_t)B.nslots, (size_t)base, O.pol}, (B.slice_ptr[O.s0 + j + 1] - base) / kSlice);
	};
	// r = b - A x with the FP32 blocks and x in global memory; this warp's part of r.M^-1 r
	auto residual = [&]() -> Fixed {
		return O.row_sum<float>([&](int j, int i) {
			const Row v = row(j, i);
			float b[3], rr[3], ss[3], qh[3], ql[3];
			vld<float, LdPlain>((const float*)B.pb, i, b);
			matrix32(j, [&](const auto& m, int w) { team_spmv_row_ff(m, w, lane, B.xff, qh, ql); });
#pragma unroll
			for (int c = 0; c < 3; ++c) rr[c] = ff_residual(b[c], qh[c], ql[c]);
			row_precond<float>(B, v.m, i, rr, ss);
			vst(v.r, 0, rr);
			return term3(rr, ss);
		});
	};
	auto publish_x = [&] {
		O.rows([&](int j, int i) {
			if (j >= O.vec_slices) return;
			float xh[3], xl[3];
			ff_ld(row(j, i).x, 0, xh, xl);
			ff_st(B.xff, i, xh, xl);
		});
	};
	const float zero[3] = {0.0f, 0.0f, 0.0f};

	O.load();
	Fixed part = O.row_sum<float>([&](int j, int i) {
		const Row v = row(j, i);
		float t[3], ss[3];
		if (j < O.vec_slices && B.precond != B3G_PRECOND_BLOCK_JACOBI)
		{
			vld<float, LdPlain>((const float*)B.Minv, i, t);
			vst(v.m, 0, t);
		}
		if (P.warm)
		{
			if (j >= O.vec_slices) return 0.0f;
			float xh[3], xl[3];
			ff_ld(B.xff, i, xh, xl);
			ff_st(v.x, 0, xh, xl);
			return 0.0f;
		}
		vld<float, LdPlain>((const float*)B.pb, i, t);
		vst(v.r, 0, t);
		vld<float, LdPlain>(sv, i, ss);
		ff_st(v.x, 0, zero, zero);
		return term3(t, ss);
	});
	if (P.warm) part = residual();
	SolveEnd S;
	S.iter = 0;
	S.delta = S.delta0 = T.sum<false>(part);
	bool done = solve_over(S.delta0, P.tol2, P.max_iter, S.status);
	double pq_prev = 0.0;
	while (!done && T.ok)
	{
		// inner solve: r, s = M^-1 r, z = 0
		++version;
		part = O.row_sum<float>([&](int j, int i) {
			const Row v = row(j, i);
			float r[3], s[3];
			vld<float, LdPlain>(v.r, 0, r);
			row_precond<float>(B, v.m, i, r, s);
			vst(v.ri, 0, r);
			store_s(i, s);
			vst(v.z, 0, zero);
			return term3(r, s);
		});
		// a warm start finds an s of any version: fenced once
		if (kVersions && P.warm && S.iter == 0) T.publish();
		double delta = T.sum<!kVersions>(part);
		if (!T.ok) break;
		float beta = 0.0f;
		if (isfinite(delta) && delta > 0.0)
			for (int it = 0; it < inner; ++it)
			{
				part = O.row_sum<float>([&](int j, int i) {
					const Row v = row(j, i);
					float o[3], dn[3];
					O.matrix(j, [&](const auto& m, int w) { team_spmv_row<TA, float, kDepth, Gather>(m, w, lane, sv, version, &sh, o, dn); });
					if (it > 0)
					{
						float dp[3], qp[3];
						vld<float, LdPlain>(v.di, 0, dp);
						vld<float, LdPlain>(v.qi, 0, qp);
#pragma unroll
						for (int c = 0; c < 3; ++c)
						{
							dn[c] = dn[c] + beta * dp[c];
							o[c] = o[c] + beta * qp[c];
						}
					}
					vst(v.qi, 0, o);
					vst(v.di, 0, dn);
					return term3(dn, o);
				});
				const double dq = T.sum<false>(part, [] {}, [&](double t) { return Divisor<float>(t).divide(delta); });
				if (!T.ok || !bits_finite(dq) || !bits_positive(dq)) break;
				const float alpha = T.ratio;
				const Divisor<float> by_delta(delta);
				++version;
				part = O.row_sum<float>([&](int j, int i) {
					const Row v = row(j, i);
					float r[3], q[3], s[3];
					vld<float, LdPlain>(v.ri, 0, r);
					vld<float, LdPlain>(v.qi, 0, q);
#pragma unroll
					for (int c = 0; c < 3; ++c) r[c] -= alpha * q[c];
					row_precond<float>(B, v.m, i, r, s);
					vst(v.ri, 0, r);
					store_s(i, s);
					return term3(r, s);
				});
				const double dn = T.sum<!kVersions>(part, [&] {
					O.rows([&](int j, int i) {
						const Row v = row(j, i);
						row_x_update<float, false>(v.z, v.di, alpha);
					});
				}, [&](double t) { return by_delta.divide(t); });
				if (!T.ok) break;
				beta = T.ratio;
				delta = dn;
				if (!bits_finite(dn) || !bits_positive(dn)) break;
			}
		if (!T.ok) break;
		// the direction p, made A-orthogonal to the previous one, in global memory for the product
		float bp = 0.0f;
		if (S.iter > 0)
		{
			part = O.row_sum<float>([&](int j, int i) {
				const Row v = row(j, i);
				float z[3], q[3];
				vld<float, LdPlain>(v.z, 0, z);
				vld<float, LdPlain>(v.q, 0, q);
				return term3(z, q);
			});
			const double gamma = T.sum<false>(part);
			if (!T.ok) break;
			bp = (float)(-gamma / pq_prev);
		}
		O.rows([&](int j, int i) {
			const Row v = row(j, i);
			float z[3];
			vld<float, LdPlain>(v.z, 0, z);
			if (S.iter > 0)
			{
				float p[3];
				vld<float, LdPlain>(v.p, 0, p);
#pragma unroll
				for (int c = 0; c < 3; ++c) z[c] = z[c] + bp * p[c];
			}
			vst(v.p, 0, z);
			vst((float*)B.d2, i, z);
		});
		T.publish();
		if (!T.ok) break;
		part = O.row_sum<float>([&](int j, int i) {
			const Row v = row(j, i);
			float o[3], p[3];
			matrix32(j, [&](const auto& m, int w) { team_spmv_row<float, float, kDepth, LdCG>(m, w, lane, pv, 0u, &sh, o, p); });
			vst(v.q, 0, o);
			return term3(p, o);
		});
		const double pq = T.sum<false>(part);
		if (!T.ok) break;
		const double pr = T.sum<false>(O.row_sum<float>([&](int j, int i) {
			const Row v = row(j, i);
			float p[3], r[3];
			vld<float, LdPlain>(v.p, 0, p);
			vld<float, LdPlain>(v.r, 0, r);
			return term3(p, r);
		}));
		if (!T.ok) break;
		pq_prev = pq;
		if (!isfinite(pq) || !isfinite(pr))
		{
			S.status = B3G_SOLVE_NONFINITE;
			break;
		}
		if (!(pq > 0.0))
		{
			S.status = B3G_SOLVE_BREAKDOWN;
			break;
		}
		const float alpha = (float)(pr / pq);
		const bool refresh = P.refresh > 0 && (S.iter % P.refresh) == 0;
		part = O.row_sum<float>([&](int j, int i) {
			const Row v = row(j, i);
			row_x_update<float, true>(v.x, v.p, alpha);
			if (refresh) return 0.0f;
			float r[3], q[3], s[3];
			vld<float, LdPlain>(v.r, 0, r);
			vld<float, LdPlain>(v.q, 0, q);
#pragma unroll
			for (int c = 0; c < 3; ++c) r[c] -= alpha * q[c];
			row_precond<float>(B, v.m, i, r, s);
			vst(v.r, 0, r);
			return term3(r, s);
		});
		if (refresh)
		{
			publish_x();
			T.publish();
			if (!T.ok) break;
			part = residual();
		}
		const double dn = T.sum<false>(part);
		S.delta = dn;
		S.iter += 1;
		if (!isfinite(dn)) S.status = B3G_SOLVE_NONFINITE;
		else if (dn <= P.tol2 * S.delta0) S.status = B3G_SOLVE_CONVERGED;
		else if (S.iter >= P.max_iter) S.status = B3G_SOLVE_MAX_ITERATIONS;
		else continue;
		break;
	}
	if (!T.ok)
	{
		team_fault(B);
		return;
	}
	if (P.newton < 0 || P.forces_left) publish_x();
	team_end(
	    T, B, P, S,
	    [&](auto f) { O.rows([&](int j, int i) { f(i, row_dv<float, true>(row(j, i).x)); }); },
	    [&](int i, float3 dv, bool finish) { return final_vertex_dv<LdPlain, FILTER>(B, i, P.h, P.newton == 0, finish, dv); });
}

} // namespace

} // namespace b3g
