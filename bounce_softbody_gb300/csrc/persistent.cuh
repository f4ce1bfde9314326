// Batch kernels: many independent bodies step in an element, a row and a solve launch per Newton
// iteration (k_batch_elements, k_batch_rows, k_batch_solve) or, with more than kFlatNewton of them, in
// one launch (k_batch).
//
// k_batch: a body is owned by a team: either a thread-block cluster of CL CTAs (large bodies) or a
// single CTA (small bodies). The team runs the whole implicit step of its body without leaving
// the kernel: element phase, row assembly, PCG, final update. Team-wide synchronisation is the
// hardware cluster barrier (or __syncthreads for one CTA); dot products are reduced per warp by
// shuffles, per CTA through shared memory and across the cluster through distributed shared
// memory, always in the same order, so every thread of the team holds the same bitwise value
// and takes the same solver decisions without a round trip to global memory. There is no
// spin-wait anywhere: the only inter-CTA waits are hardware barriers between CTAs that the
// cluster launch guarantees to be co-resident.
//
// Work distribution: bodies are sorted by size (largest first). Clusters first take large bodies
// from a global counter; when those run out every CTA takes small bodies on its own.
//
// k_batch_solve: the solve of solve.cuh by teams of a cluster or of the half, quarter, ... of one, each
// width taking its bodies from its own counter, widest first.
//
// This header holds the kernel templates; persistent_{f32,f64,bf16}.cu instantiate one
// precision each (compiled in parallel) and persistent.cu dispatches.
#pragma once

#include "device.cuh"
#include "ops.h"
#include "solve.cuh"

#include <atomic>
#include <cooperative_groups.h>
#include <type_traits>
#include <utility>

namespace cg = cooperative_groups;

namespace b3g {

struct BatchParams
{
	const DevBody* bodies;
	const int* big;
	int nbig;
	const int* small;
	int nsmall;
	unsigned* queue;
	int solve_ctas;        // CTAs of the solve launch (0: as many clusters as fit)
	int polls;             // of a solve team's wait before it gives up, 0: the default
	int tier_end[kTiers];  // of the order `big` (which runs on into `small`): the solve launch's teams
	int steps;
	float h;
	int newton;
	int k;                 // flat: the Newton iteration of these launches
	int max_iter;
	double tol2;
	int refresh;
	double newton_tol2;
	unsigned long long* prof;  // optional: kPhases cycle counters per CTA
	// flat: a Newton iteration's elements and rows run in the flat launches (their numbering below)
	int flat;
	const unsigned* elem_off;
	const unsigned* slice_off;
	unsigned nelem;
	unsigned nslices;
	int nbodies;
	int tets_only;   // every body: tetrahedra only, no contact spheres (the row assembly's short form)
	int filter;      // filtered contacts: bodies with a constraint buffer (filt) are stepped in that mode
	// flat launches over part of the numbering: elements [g_begin, nelem), slices [s_begin,
	// nslices); rows_per_sm > 0 caps the row launch at that many CTAs per SM (0: all resident)
	unsigned g_begin;
	unsigned s_begin;
	int rows_per_sm;
};

namespace {

// resident CTAs per SM the team assembly's register budget is sized for (128 registers a thread)
#ifndef B3G_BATCH_MIN_BLOCKS
#define B3G_BATCH_MIN_BLOCKS (B3G_PCG_THREADS >= 512 ? 1 : 2)
#endif

constexpr int kPThreads = B3G_PCG_THREADS;  // ops.h
constexpr int kPWarps = kPThreads / 32;

struct TeamShared
{
	double wp[2][kPWarps];
	double slot[2];
	int item;
	int pad;
};

template <int CL>
struct Team
{
	TeamShared* sh;
	int parity;
	int rank;

	__device__ void sync()
	{
		if (CL == 1) __syncthreads();
		else cg::this_cluster().sync();
	}
	__device__ int tid() const { return rank * kPThreads + (int)threadIdx.x; }
	__device__ int nthreads() const { return CL * kPThreads; }
	__device__ int warp() const { return rank * kPWarps + ((int)threadIdx.x >> 5); }
	__device__ int nwarps() const { return CL * kPWarps; }

	// Team-wide sum; every thread of the team returns the same value (fixed summation order).
	__device__ double reduce(double v)
	{
		const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
		v = warp_sum(v);
		if (lane == 0) sh->wp[parity][w] = v;
		__syncthreads();
		double t = 0.0;
#pragma unroll
		for (int k = 0; k < kPWarps; ++k) t += sh->wp[parity][k];
		if (CL > 1)
		{
			if (threadIdx.x == 0) sh->slot[parity] = t;
			cg::cluster_group cl = cg::this_cluster();
			cl.sync();
			double u = 0.0;
			if (lane < CL) u = *cl.map_shared_rank(&sh->slot[parity], lane);
			t = warp_sum(u);
		}
		parity ^= 1;
		return t;
	}
};


struct PhaseClock
{
	unsigned long long* slot;
	long long t;
	__device__ void start(unsigned long long* p)
	{
		slot = p ? p + (size_t)blockIdx.x * kPhases : nullptr;
		if (slot) t = clock64();
	}
	__device__ void tick(int phase)
	{
		if (!slot) return;
		long long now = clock64();
		// (atomic: a CTA of a second solve launch shares the slot of its block id)
		if (threadIdx.x == 0) atomicAdd(slot + phase, (unsigned long long)(now - t));
		t = now;
	}
};

// PCG update of row i: x += alpha d and, unless this is a refresh iteration, r -= alpha q, s = M^-1 r.
// Returns the row's r.s.
template <class TV, class LD>
__device__ __forceinline__ double update_row(const DevBody& B, TV* __restrict__ py, const TV* __restrict__ d,
                                             TV* __restrict__ r, const TV* __restrict__ q, TV* __restrict__ s, int i,
                                             TV alpha, bool refresh)
{
	TV x[3], dd[3], rr[3], qq[3];
	vld<TV, LD>(py, i, x);
	vld<TV, LD>(d, i, dd);
	if (!refresh)
	{
		vld<TV, LD>(r, i, rr);
		vld<TV, LD>(q, i, qq);
	}
#pragma unroll
	for (int c = 0; c < 3; ++c) x[c] += alpha * dd[c];
	vst(py, i, x);
	if (refresh) return 0.0;
	TV ss[3];
#pragma unroll
	for (int c = 0; c < 3; ++c) rr[c] -= alpha * qq[c];
	precond_row<TV, LD>(B, i, rr, ss);
	vst(r, i, rr);
	vst(s, i, ss);
	return dot3<TV>(rr, ss);
}

// r = pb - A x, s = M^-1 r for the rows of one warp's slices (init / refresh); optionally d = s
template <class TA, class TV, class LD>
__device__ __forceinline__ double residual_rows(const DevBody& B, const TA* A, const TV* x, int s0, int stride,
                                                bool set_d)
{
	const int lane = threadIdx.x & 31;
	double part = 0.0;
	for (int sl = s0; sl < B.nslices; sl += stride)
	{
		const int i = sl * kSlice + lane;
		if (i >= B.n) continue;
		const int base = B.slice_ptr[sl], w = (B.slice_ptr[sl + 1] - base) / kSlice;
		TV o[3], b[3], rr[3], ss[3];
		spmv_row<TA, TV, LD, MatVia<LD>>(A, B.col, B.nslots, base, w, lane, x, o);
		vld<TV, LD>((const TV*)B.pb, i, b);
#pragma unroll
		for (int c = 0; c < 3; ++c) rr[c] = b[c] - o[c];
		precond_row<TV, LD>(B, i, rr, ss);
		vst((TV*)B.r, i, rr);
		vst((TV*)B.s, i, ss);
		if (set_d) vst((TV*)B.d, i, ss);
		part += dot3<TV>(rr, ss);
	}
	return part;
}

// The direction and A times it by linearity, for the rows of one warp's slices: d = s + beta d
// and q = A s + beta q (d = s, q = A s on a solve's first iteration), and this warp's part of
// d.q. The SpMV gathers only s, which the update sweep finished before its reduction (a team
// barrier), so no direction sweep and no barrier of its own precede it. d and q stay row-local.
template <class TA, class TV, class LD>
__device__ __forceinline__ double spmv_lin_rows(const DevBody& B, const TA* A, const TV* s, TV* d, TV* q, TV beta,
                                                bool first, int s0, int stride)
{
	const int lane = threadIdx.x & 31;
	double part = 0.0;
	for (int sl = s0; sl < B.nslices; sl += stride)
	{
		const int i = sl * kSlice + lane;
		if (i >= B.n) continue;
		const int base = B.slice_ptr[sl], w = (B.slice_ptr[sl + 1] - base) / kSlice;
		TV o[3], dd[3];
		spmv_row<TA, TV, LD, MatVia<LD>>(A, B.col, B.nslots, base, w, lane, s, o);
		vld<TV, LD>(s, i, dd);
		if (!first)
		{
			TV dp[3], qp[3];
			vld<TV, LD>(d, i, dp);
			vld<TV, LD>(q, i, qp);
#pragma unroll
			for (int c = 0; c < 3; ++c)
			{
				dd[c] = dd[c] + beta * dp[c];
				o[c] = o[c] + beta * qp[c];
			}
		}
		vst(q, i, o);
		vst(d, i, dd);
		part += dot3<TV>(dd, o);
	}
	return part;
}

// Filtered-contact forms of the row assembly and of the final update, out of line so that the
// default forms inlined in the team kernels keep their register allocation.
template <class TA, class TV, class LD>
__device__ __noinline__ double assemble_row_filtered(const DevBody& B, int sl, int lane, const StepParams& sp,
                                                     int init)
{
	return assemble_row<TA, TV, LD, true>(B, sl, lane, sp, init);
}

__device__ __noinline__ void contact_filter_vertex_ool(const DevBody& B, int i, float h)
{
	contact_filter_vertex(B, i, h);
}

template <class TV, class LD>
__device__ __noinline__ double final_vertex_filtered(const DevBody& B, int i, float h, bool first, bool finish)
{
	return final_vertex<TV, LD, true>(B, i, h, first, finish);
}

// Result of one PCG solve of a team.
struct SolveOut
{
	int iter;
	int status;
	double delta;
};

// The preconditioned CG of one body by one team, from r, s, d, py set up by the assembly (or a
// warm start) with r.s = delta0 (sparse_solver.cpp:57-108 with the true-residual refresh).
template <int CL, class TA, class TV, class LD>
__device__ SolveOut team_pcg(Team<CL>& T, const DevBody& B, const BatchParams& P, bool bf16, double delta0,
                             PhaseClock& pc)
{
	const int lane = threadIdx.x & 31;
	const TA* Asp = (sizeof(TA) == sizeof(float) && !bf16) ? (const TA*)B.A32 : (const TA*)B.Alo;
	TV* py = (TV*)B.py;
	TV* r = (TV*)B.r;
	TV* s = (TV*)B.s;
	TV* d = (TV*)B.d;
	TV* q = (TV*)B.q;
	SolveOut out;
	out.status = B3G_SOLVE_CONVERGED;
	out.iter = 0;
	double delta = delta0;
	bool pending = false;
	bool done;
	if (!isfinite(delta0))
	{
		out.status = B3G_SOLVE_NONFINITE;
		done = true;
	}
	else if (delta0 <= P.tol2 * delta0)
	{
		out.status = B3G_SOLVE_CONVERGED;
		done = true;
	}
	else if (P.max_iter <= 0)
	{
		out.status = B3G_SOLVE_MAX_ITERATIONS;
		done = true;
	}
	else
		done = false;
	int iter = 0;
	TV bt = (TV)0;
	while (!done)
	{
		// d = s + beta d, q = A d (as A s + beta q), alpha = delta / d.q
		double part = spmv_lin_rows<TA, TV, LD>(B, Asp, s, d, q, bt, iter == 0, T.warp(), T.nwarps());
		const double dq = T.reduce(part);
		pc.tick(kPhSpmv);
		if (!isfinite(dq))
		{
			out.status = B3G_SOLVE_NONFINITE;
			break;
		}
		if (!(dq > 0.0))
		{
			out.status = B3G_SOLVE_BREAKDOWN;
			break;
		}
		const TV alpha = (TV)(delta / dq);
		const bool refresh = (P.refresh > 0 && (iter % P.refresh) == 0) || pending;
		part = 0.0;
		for (int sl = T.warp(); sl < B.nslices; sl += T.nwarps())
		{
			const int i0 = sl * kSlice + lane;
			if (i0 >= B.n) continue;
			part += update_row<TV, LD>(B, py, d, r, q, s, i0, alpha, refresh);
		}
		if (refresh)
		{
			// sparse_solver.cpp:83-90: r = b - A x with the full-precision blocks
			T.sync();
			part = (sizeof(TA) == sizeof(double))
			           ? residual_rows<TA, TV, LD>(B, Asp, py, T.warp(), T.nwarps(), false)
			           : residual_rows<float, TV, LD>(B, B.A32, py, T.warp(), T.nwarps(), false);
		}
		const double dn = T.reduce(part);
		pc.tick(kPhUpdate);
		const double beta = dn / delta;
		delta = dn;
		iter += 1;
		if (!isfinite(dn))
		{
			out.status = B3G_SOLVE_NONFINITE;
			break;
		}
		bool conv = dn <= P.tol2 * delta0;
		if (bf16 && conv && !refresh)
		{
			pending = true;
			conv = false;
		}
		if (refresh) pending = false;
		if (conv)
		{
			out.status = B3G_SOLVE_CONVERGED;
			break;
		}
		if (iter >= P.max_iter)
		{
			out.status = B3G_SOLVE_MAX_ITERATIONS;
			break;
		}
		bt = (TV)beta;
	}
	out.iter = iter;
	out.delta = delta;
	return out;
}

// Element phase and row assembly of one Newton iteration; returns the team's r.s (the PCG's
// delta0). k > 0 warm-starts from the previous solution: r = pb - A py.
template <int CL, class TA, class TV, class LD>
__device__ double team_assemble(Team<CL>& T, const DevBody& B, const BatchParams& P, bool bf16, int k, PhaseClock& pc)
{
	const int lane = threadIdx.x & 31;
	StepParams sp;
	sp.h = P.h;
	sp.first_newton = k == 0 ? 1 : 0;
	if (k == 0 && B.filt)
	{
		// filtered contacts: the contact update and each vertex's constraint at the step's start
		for (int i = T.tid(); i < B.n; i += T.nthreads()) contact_filter_vertex_ool(B, i, P.h);
		T.sync();
	}
	for (int e = T.tid(); e < B.nt; e += T.nthreads()) tet_element<LD>(B, e, sp);
	for (int e = T.tid(); e < B.ntr; e += T.nthreads()) tri_element<LD>(B, e, sp);
	for (int e = T.tid(); e < B.ns; e += T.nthreads()) spring_element<LD>(B, e, sp);
	for (int e = T.tid(); e < B.nbw; e += T.nthreads()) bw_element<LD>(B, e, sp);
	for (int e = T.tid(); e < B.nms; e += T.nthreads()) mouse_element<LD>(B, e, sp);
	T.sync();
	pc.tick(kPhElem);
	double part = 0.0;
	for (int sl = T.warp(); sl < B.nslices; sl += T.nwarps())
		part += B.filt ? assemble_row_filtered<TA, TV, LD>(B, sl, lane, sp, k == 0 ? kInitAll : kInitNone)
		               : assemble_row<TA, TV, LD>(B, sl, lane, sp, k == 0 ? kInitAll : kInitNone);
	if (k > 0)
	{
		const TA* Asp = (sizeof(TA) == sizeof(float) && !bf16) ? (const TA*)B.A32 : (const TA*)B.Alo;
		T.sync();
		part = (sizeof(TA) == sizeof(double))
		           ? residual_rows<TA, TV, LD>(B, Asp, (const TV*)B.py, T.warp(), T.nwarps(), true)
		           : residual_rows<float, TV, LD>(B, B.A32, (const TV*)B.py, T.warp(), T.nwarps(), true);
	}
	const double delta0 = T.reduce(part);
	pc.tick(kPhAsm);
	return delta0;
}

// Final update of a single-Newton step (state, friction, clearing, new contacts) and the
// step's statistics.
template <int CL, class TV, class LD>
__device__ void team_finish(Team<CL>& T, const DevBody& B, const BatchParams& P, const SolveOut& so, double delta0,
                            int newton_iters, int min_it, int max_it, unsigned long long iters_all, double err,
                            PhaseClock& pc)
{
	T.sync();
	if (T.tid() == 0)
	{
		Scalars* sc = B.sc;
		sc->iter = so.iter;
		sc->delta = so.delta;
		sc->delta0 = delta0;
		sc->status = so.status;
		sc->min_it = min_it;
		sc->max_it = max_it;
		sc->newton_iter = newton_iters;
		sc->newton_err = err;
		sc->pending = 0;
		if (sc->fault) sc->status = B3G_SOLVE_DEVICE_TIMEOUT;
		sc->total_iters += iters_all;
		sc->total_steps += 1ull;
	}
}

// The whole implicit step of one body by one team (any number of Newton iterations); mirrors
// the single-body step phase for phase (same device functions, same solver decisions).
template <int CL, class TA, class TV>
__device__ void team_step(Team<CL>& T, const DevBody& B, const BatchParams& P, bool bf16)
{
	// A single-CTA team reads what its own threads wrote behind __syncthreads: ordinary (L1)
	// loads are coherent there. Cluster teams read other SMs' writes: L2-coherent loads.
	typedef typename std::conditional<CL == 1, LdPlain, LdCG>::type LD;
	const int lane = threadIdx.x & 31;
	const float h = P.h;
	int min_it = 0x7fffffff, max_it = 0, newton_done_at = 0;
	double delta0 = 0.0, err = 0.0, err0 = 0.0;
	unsigned long long iters_all = 0ull;
	SolveOut so;
	so.iter = 0;
	so.status = B3G_SOLVE_CONVERGED;
	so.delta = 0.0;
	PhaseClock pc;
	pc.start(P.prof);
	if (T.tid() == 0) B.sc->fault = 0;  // ordered before any SpMV by the element-phase barrier
	for (int k = 0; k < P.newton; ++k)
	{
		const bool finish = P.newton == 1;
		delta0 = team_assemble<CL, TA, TV, LD>(T, B, P, bf16, k, pc);
		so = team_pcg<CL, TA, TV, LD>(T, B, P, bf16, delta0, pc);
		min_it = so.iter < min_it ? so.iter : min_it;
		max_it = so.iter > max_it ? so.iter : max_it;
		iters_all += (unsigned long long)so.iter;
		// every thread finished its PCG reads before the final update rewrites x / v
		T.sync();
		double part = 0.0;
		for (int sl = T.warp(); sl < B.nslices; sl += T.nwarps())
		{
			const int i = sl * kSlice + lane;
			if (i < B.n)
				part += B.filt ? final_vertex_filtered<TV, LD>(B, i, h, k == 0, finish)
				               : final_vertex<TV, LD>(B, i, h, k == 0, finish);
		}
		err = T.reduce(part);
		pc.tick(kPhFinal);
		if (k == 0) err0 = err;
		newton_done_at = k + 1;
		if (finish) break;
		const bool ndone = k == 0 ? err <= P.newton_tol2 : err <= P.newton_tol2 * err0;
		if (ndone || k == P.newton - 1)
		{
			T.sync();
			for (int sl = T.warp(); sl < B.nslices; sl += T.nwarps())
			{
				const int i = sl * kSlice + lane;
				if (i < B.n) post_vertex<LD>(B, i, h);
			}
			break;
		}
	}
	team_finish<CL, TV, LD>(T, B, P, so, delta0, newton_done_at, min_it, max_it, iters_all, err, pc);
}

// Single-Newton step split in two launches so that each part runs with its own register budget
// (one CTA per SM for the solve, several for the assembly). Part 1: elements and assembly; k_batch_solve
// does the rest.
template <int CL, class TA, class TV>
__device__ void team_step_assemble(Team<CL>& T, const DevBody& B, const BatchParams& P, bool bf16)
{
	typedef typename std::conditional<CL == 1, LdPlain, LdCG>::type LD;
	PhaseClock pc;
	pc.start(P.prof);
	if (T.tid() == 0) solve_pending(B, true);
	team_assemble<CL, TA, TV, LD>(T, B, P, bf16, 0, pc);
}

__device__ void load_body(DevBody* dst, const DevBody* src)
{
	const int words = (int)(sizeof(DevBody) / sizeof(int));
	const int* s = (const int*)src;
	int* d = (int*)dst;
	for (int k = threadIdx.x; k < words; k += blockDim.x) d[k] = __ldcg(s + k);
}

// Launch phases of the team kernel: the whole step (any number of Newton iterations), or the
// assembly of a single-Newton step, which k_batch_solve completes from its own pair of counters.
enum { kPhaseWhole = 0, kPhaseAssemble = 1 };

template <int CL, class TA, class TV, int PH>
__device__ __forceinline__ void team_run(Team<CL>& T, const DevBody& B, const BatchParams& P, bool bf16)
{
	if (PH == kPhaseWhole) team_step<CL, TA, TV>(T, B, P, bf16);
	else team_step_assemble<CL, TA, TV>(T, B, P, bf16);
}

template <int CL, class TA, class TV, int PH>
__global__ void __launch_bounds__(kPThreads, B3G_BATCH_MIN_BLOCKS) k_batch(BatchParams P, int bf16)
{
	__shared__ TeamShared sh;
	__shared__ __align__(16) DevBody sb;
	unsigned* queue = P.queue;

	if (CL > 1)
	{
		cg::cluster_group cl = cg::this_cluster();
		Team<CL> T;
		T.sh = &sh;
		T.parity = 0;
		T.rank = (int)cl.block_rank();
		for (;;)
		{
			if (T.rank == 0 && threadIdx.x == 0) sh.item = (int)atomicAdd(queue, 1u);
			cl.sync();
			const int item = *cl.map_shared_rank(&sh.item, 0);
			cl.sync();
			if (item >= P.nbig) break;
			load_body(&sb, P.bodies + P.big[item]);
			__syncthreads();
			for (int st = 0; st < P.steps; ++st) team_run<CL, TA, TV, PH>(T, sb, P, bf16 != 0);
			cl.sync();
		}
	}
	Team<1> T1;
	T1.sh = &sh;
	T1.parity = 0;
	T1.rank = 0;
	for (;;)
	{
		if (threadIdx.x == 0) sh.item = (int)atomicAdd(queue + 1, 1u);
		__syncthreads();
		const int item = sh.item;
		__syncthreads();
		if (item >= P.nsmall) break;
		load_body(&sb, P.bodies + P.small[item]);
		__syncthreads();
		for (int st = 0; st < P.steps; ++st) team_run<1, TA, TV, PH>(T1, sb, P, bf16 != 0);
		__syncthreads();
	}
}

// The PCG, the final update and the statistics of every body of a batch, one Newton iteration. A body's
// team is a cluster or an aligned half, quarter ... of one (its tier); each body is solved by
// team_solve with its rows' vectors and as much of its matrix as fits in shared memory.
// One CTA of 512 threads per SM (128 registers a thread, the SM's shared memory to itself). Measured
// on 160 / 12 uneven blocks and 16 blocks and cloths, ms a step: 512 x 1 12.1 / 1.54 / 7.0, 640 x 1
// 12.2 / 1.59 / 6.6, 768 x 1 14.4 / 1.68 / 7.4 (spills), 320 x 2 12.9 / 1.90 / 8.8, 256 x 2 14.5 /
// 1.97 / 10.8; the launch before (256 x 4, every vector and matrix through L2 and HBM) 14.0 / 2.99 / 12.1.

__device__ __noinline__ double final_vertex_dv_filtered(const DevBody& B, int i, float h, bool first, bool finish, float3 dv)
{
	return final_vertex_dv<LdPlain, true>(B, i, h, first, finish, dv);
}

template <class TA, class TV, class Team>
__device__ __forceinline__ void batch_solve_body(Team& T, const DevBody& B, const BatchParams& P, unsigned char* smem, int room)
{
	PhaseClock pc;
	pc.start(P.prof);
	SolveArgs A;
	A.tol2 = P.tol2;
	A.newton_tol2 = P.newton_tol2;
	A.max_iter = P.max_iter;
	A.refresh = P.refresh;
	A.h = P.h;
	A.newton = P.k;
	A.newton_max = P.newton;
	A.forces_left = P.k + 1 < P.newton ? 1 : 0;
	A.warm = P.k > 0 ? 1 : 0;
	A.smem = room;
	A.keep = 1024;
	A.polls = P.polls;
	team_solve<TA, TV, false, 1>(
	    T, B, A, smem,
	    [&](int i, float3 dv, bool finish) {
		    return B.filt ? final_vertex_dv_filtered(B, i, A.h, A.newton == 0, finish, dv)
		                  : final_vertex_dv<LdPlain, false>(B, i, A.h, A.newton == 0, finish, dv);
	    },
	    [&](int phase) { pc.tick(phase); });
}

template <class TA, class TV>
__global__ void __launch_bounds__(kSolveMaxThreads, 1) k_batch_solve(BatchParams P, int room)
{
	extern __shared__ __align__(16) unsigned char smem[];
	__shared__ SolveSh sh;
	__shared__ __align__(16) DevBody sb;
	cg::cluster_group cl = cg::this_cluster();
	ClusterTeam<TV> T(&sh, P.polls);
	cl.sync();
	// widest teams first; a cluster whose wider teams find no more bodies splits into narrower ones.
	// A CTA one of whose waits ran out takes part in no further sum: its teammates run out at their next
	// one, so no partial of one sum is taken for another's, and the bodies they leave are reported.
	int begin = 0;
	for (int t = 0; t < kTiers && T.ok; ++t)
	{
		const int end = P.tier_end[t], width = kMaxTeamCtas >> t;
		if (end > begin && width <= (int)cl.num_blocks())
		{
			T.form(width);
			for (;;)
			{
				// the next body whose Newton loop goes on (the team's first thread decides for all)
				int taken = end;
				const int item = begin + T.agree([&] {
					do
					{
						taken = begin + (int)min(atomicAdd(P.queue + 2 + t, 1u), 1u << 28);
					} while (taken < end && P.k > 0 && P.bodies[P.big[taken]].sc->newton_done);
					return taken - begin;
				});
				if (!T.ok && taken < end) team_fault(P.bodies[P.big[taken]]);
				if (!T.ok || item < begin || item >= end) break;
				load_body(&sb, P.bodies + P.big[item]);
				__syncthreads();
				batch_solve_body<TA, TV>(T, sb, P, smem, room);
				if (!T.ok) break;
			}
		}
		begin = end;
	}
	cl.sync();
}

// Clusters of more than 8 CTAs are a non-portable size the kernel has to opt in to.
template <int CL, class TA, class TV, int PH>
cudaError_t allow_cluster()
{
	if (CL <= 8) return cudaSuccess;
	return cudaFuncSetAttribute(k_batch<CL, TA, TV, PH>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}

template <int CL, class TA, class TV, int PH>
cudaError_t launch_ph(const BatchParams& P, int ctas, int bf16, cudaStream_t st)
{
	cudaError_t e = allow_cluster<CL, TA, TV, PH>();
	if (e != cudaSuccess) return e;
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3((unsigned)ctas, 1, 1);
	cfg.blockDim = dim3(kPThreads, 1, 1);
	cfg.dynamicSmemBytes = 0;
	cfg.stream = st;
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeClusterDimension;
	attr[0].val.clusterDim.x = CL;
	attr[0].val.clusterDim.y = 1;
	attr[0].val.clusterDim.z = 1;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	return cudaLaunchKernelEx(&cfg, k_batch<CL, TA, TV, PH>, P, bf16);
}

template <int CL, class TA, class TV, int PH>
int max_clusters_ph()
{
	if (allow_cluster<CL, TA, TV, PH>() != cudaSuccess) return 0;
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3(CL * 64, 1, 1);
	cfg.blockDim = dim3(kPThreads, 1, 1);
	cfg.dynamicSmemBytes = 0;
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeClusterDimension;
	attr[0].val.clusterDim.x = CL;
	attr[0].val.clusterDim.y = 1;
	attr[0].val.clusterDim.z = 1;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	int n = 0;
	if (cudaOccupancyMaxActiveClusters(&n, k_batch<CL, TA, TV, PH>, &cfg) != cudaSuccess) return 0;
	return n;
}

// Shared memory of a CTA of the solve launch: what its static part leaves of its share of the SM.
inline int solve_room()
{
	static const int room = [] {
		int dev = 0, block = 0, sm = 0;
		cudaGetDevice(&dev);
		cudaDeviceGetAttribute(&block, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
		cudaDeviceGetAttribute(&sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
		return (std::min(block, sm - 1024) - (int)(sizeof(SolveSh) + sizeof(DevBody)) - 256 - kL1Room) & ~127;
	}();
	return room;
}

template <class TA, class TV>
cudaError_t solve_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, int cluster, int ctas, cudaStream_t st)
{
	cudaError_t e = cudaFuncSetAttribute(k_batch_solve<TA, TV>, cudaFuncAttributeMaxDynamicSharedMemorySize, solve_room());
	if (e == cudaSuccess && cluster > 8)
		e = cudaFuncSetAttribute(k_batch_solve<TA, TV>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
	*cfg = {};
	cfg->gridDim = dim3((unsigned)ctas, 1, 1);
	cfg->blockDim = dim3(kSolveMaxThreads, 1, 1);
	cfg->dynamicSmemBytes = (size_t)solve_room();
	cfg->stream = st;
	attr->id = cudaLaunchAttributeClusterDimension;
	attr->val.clusterDim.x = (unsigned)cluster;
	attr->val.clusterDim.y = 1;
	attr->val.clusterDim.z = 1;
	cfg->attrs = attr;
	cfg->numAttrs = 1;
	return e;
}

// Co-resident clusters of the solve launch, queried once per precision and cluster size.
template <class TA, class TV>
int solve_clusters(int cluster)
{
	static std::atomic<int> cached[kMaxTeamCtas + 1];  // count + 1; 0: not known yet
	int m = cached[cluster].load(std::memory_order_relaxed) - 1;
	if (m < 0)
	{
		cudaLaunchConfig_t cfg;
		cudaLaunchAttribute attr;
		m = 0;
		if (solve_config<TA, TV>(&cfg, &attr, cluster, cluster, nullptr) == cudaSuccess &&
		    cudaOccupancyMaxActiveClusters(&m, k_batch_solve<TA, TV>, &cfg) != cudaSuccess)
			m = 0;
		cudaGetLastError();
		cached[cluster].store(m + 1, std::memory_order_relaxed);
	}
	return m;
}

// One step: the whole-step kernel for many Newton iterations, else the assembly launch
// (`ctas` CTAs) followed by the solve launch (as many CTAs as fit). part 1 / 2 issues only the
// assembly / solve launch of a single-Newton step (timed separately), 0 both.
template <int CL, class TA, class TV>
cudaError_t launch_cl(const BatchParams& P, int ctas, int bf16, int part, cudaStream_t st)
{
	if (P.newton > 1 && !P.flat) return launch_ph<CL, TA, TV, kPhaseWhole>(P, ctas, bf16, st);
	if (part != 2 && !P.flat)
	{
		cudaError_t e = launch_ph<CL, TA, TV, kPhaseAssemble>(P, ctas, bf16, st);
		if (e != cudaSuccess || part == 1) return e;
	}
	const int m = solve_clusters<TA, TV>(CL);
	cudaLaunchConfig_t cfg;
	cudaLaunchAttribute attr;
	cudaError_t e = solve_config<TA, TV>(&cfg, &attr, CL, P.solve_ctas > 0 ? P.solve_ctas : (m > 0 ? m * CL : CL), st);
	if (e != cudaSuccess) return e;
	return cudaLaunchKernelEx(&cfg, k_batch_solve<TA, TV>, P, solve_room());
}

// The body of flat item g: the last k with off[k] <= g.
__device__ __forceinline__ int flat_body(const unsigned* __restrict__ off, int nbodies, unsigned g)
{
	int lo = 0, hi = nbodies - 1;
	while (lo < hi)
	{
		const int mid = (lo + hi + 1) >> 1;
		if (__ldg(off + mid) <= g) lo = mid;
		else hi = mid - 1;
	}
	return lo;
}

// The row assembly of every body of a batch, one warp per slice over a flat numbering of all
// bodies' slices: no team, no barrier, and the load spreads evenly over the GPU whatever the
// bodies' sizes (the team launch's tail was set by its largest bodies). Element records come from
// the flat element launch before it, state from earlier launches: plain loads. The PCG launch
// sums delta0 = r.s per body itself.
#ifndef B3G_ROWS_THREADS
#define B3G_ROWS_THREADS 256     // threads per CTA of the flat row launch
#endif
#ifndef B3G_ROWS_MIN_BLOCKS
#define B3G_ROWS_MIN_BLOCKS 2    // resident CTAs per SM its register budget is sized for
#endif
constexpr int kRowsWarps = B3G_ROWS_THREADS / 32;

#ifndef B3G_ROWS_TETS_MIN_BLOCKS
#define B3G_ROWS_TETS_MIN_BLOCKS 3  // the tetrahedra-only row assembly fits more CTAs per SM
#endif

// FILT: some bodies have filtered contacts (their filt buffer set); each body takes its own form.
// LATER: a Newton iteration after the first (a form of its own keeps the first one's registers).
template <class TA, class TV, bool TETS, bool FILT, bool LATER>
__global__ void __launch_bounds__(B3G_ROWS_THREADS, TETS ? B3G_ROWS_TETS_MIN_BLOCKS : B3G_ROWS_MIN_BLOCKS)
k_batch_rows(BatchParams P)
{
	// each warp's body descriptor, copied to shared memory: the row code's stores to global
	// memory cannot alias it there, so its fields need not be re-read after each store
	static_assert(sizeof(DevBody) % 8 == 0, "DevBody is copied in 8-byte words");
	__shared__ DevBody s_body[kRowsWarps];
	const int lane = threadIdx.x & 31;
	DevBody& B = s_body[threadIdx.x >> 5];
	StepParams sp;
	sp.h = P.h;
	sp.first_newton = LATER ? 0 : 1;
	const int init = LATER ? kInitNone : kInitTeam;
	const unsigned nw = gridDim.x * kRowsWarps;
	for (unsigned g = P.s_begin + blockIdx.x * kRowsWarps + (threadIdx.x >> 5); g < P.nslices; g += nw)
	{
		const int b = flat_body(P.slice_off, P.nbodies, g);
		__syncwarp();
		{
			const unsigned long long* src = reinterpret_cast<const unsigned long long*>(P.bodies + b);
			unsigned long long* dst = reinterpret_cast<unsigned long long*>(&B);
			for (int w = lane; w < (int)(sizeof(DevBody) / 8); w += 32) dst[w] = __ldg(src + w);
		}
		__syncwarp();
		if (LATER && B.sc->newton_done) continue;
		const int sl = (int)(g - __ldg(P.slice_off + b));
		if (sl == 0 && lane == 0) solve_pending(B, !LATER);
		if (FILT && B.filt) assemble_row_filtered<TA, TV, LdPlain>(B, sl, lane, sp, init);
		else assemble_row<TA, TV, LdPlain, false, TETS>(B, sl, lane, sp, init);
	}
}

template <class TA, class TV, bool TETS, bool FILT, bool LATER>
cudaError_t launch_rows_t(const BatchParams& P, cudaStream_t st)
{
	static const std::pair<int, int> resident = [] {  // SMs, resident CTAs per SM
		int dev = 0, sms = 0, per_sm = 0;
		cudaGetDevice(&dev);
		cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
		cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch_rows<TA, TV, TETS, FILT, LATER>, B3G_ROWS_THREADS, 0);
		return std::make_pair(std::max(1, sms), std::max(per_sm, 1));
	}();
	const int cap = resident.first * (P.rows_per_sm > 0 ? std::min(P.rows_per_sm, resident.second) : resident.second);
	const unsigned need = (P.nslices - P.s_begin + kRowsWarps - 1) / kRowsWarps;
	const int grid = (int)std::max(1u, std::min(need, (unsigned)cap));
	k_batch_rows<TA, TV, TETS, FILT, LATER><<<grid, B3G_ROWS_THREADS, 0, st>>>(P);
	return cudaGetLastError();
}

// the tetrahedra-only kernel when every body of the batch qualifies (P.tets_only), the kernel
// with both row forms when some body has filtered contacts (P.filter)
template <class TA, class TV, bool LATER>
cudaError_t launch_rows_k(const BatchParams& P, cudaStream_t st)
{
	if (P.filter) return launch_rows_t<TA, TV, false, true, LATER>(P, st);
	return P.tets_only ? launch_rows_t<TA, TV, true, false, LATER>(P, st) : launch_rows_t<TA, TV, false, false, LATER>(P, st);
}

template <class TA, class TV>
cudaError_t launch_rows(const BatchParams& P, cudaStream_t st)
{
	return P.k > 0 ? launch_rows_k<TA, TV, true>(P, st) : launch_rows_k<TA, TV, false>(P, st);
}

template <class TA, class TV>
cudaError_t launch_prec(const BatchParams& P, int cluster, int ctas, int bf16, int part, cudaStream_t st)
{
	switch (cluster)
	{
	case 1: return launch_cl<1, TA, TV>(P, ctas, bf16, part, st);
	case 2: return launch_cl<2, TA, TV>(P, ctas, bf16, part, st);
	case 4: return launch_cl<4, TA, TV>(P, ctas, bf16, part, st);
	case 8: return launch_cl<8, TA, TV>(P, ctas, bf16, part, st);
	case 16: return launch_cl<16, TA, TV>(P, ctas, bf16, part, st);
	default: return cudaErrorInvalidValue;
	}
}

// Co-resident clusters of the assembly (and whole-step) launch; also primes the solve launch's
// count so that no occupancy query happens while a stream is being captured.
template <int CL, class TA, class TV>
int max_clusters()
{
	if (solve_clusters<TA, TV>(CL) <= 0) return 0;
	return max_clusters_ph<CL, TA, TV, kPhaseAssemble>();
}

template <class TA, class TV>
int max_clusters_prec(int cluster)
{
	switch (cluster)
	{
	case 1: return max_clusters<1, TA, TV>();
	case 2: return max_clusters<2, TA, TV>();
	case 4: return max_clusters<4, TA, TV>();
	case 8: return max_clusters<8, TA, TV>();
	case 16: return max_clusters<16, TA, TV>();
	default: return 0;
	}
}

} // namespace

// per-precision entry points (persistent_f32.cu, persistent_f64.cu, persistent_bf16.cu)
cudaError_t launch_batch_f32(const BatchParams& P, int cluster, int ctas, int part, cudaStream_t st);
cudaError_t launch_batch_f64(const BatchParams& P, int cluster, int ctas, int part, cudaStream_t st);
cudaError_t launch_batch_bf16(const BatchParams& P, int cluster, int ctas, int part, cudaStream_t st);
cudaError_t launch_rows_f32(const BatchParams& P, cudaStream_t st);
cudaError_t launch_rows_f64(const BatchParams& P, cudaStream_t st);
cudaError_t launch_rows_bf16(const BatchParams& P, cudaStream_t st);
// co-resident clusters of the solve launch
int solve_clusters_f32(int cluster);
int solve_clusters_f64(int cluster);
int solve_clusters_bf16(int cluster);
int max_clusters_f32(int cluster);
int max_clusters_f64(int cluster);
int max_clusters_bf16(int cluster);

} // namespace b3g
