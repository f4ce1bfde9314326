// Host-callable launchers of the single-body kernels (kernels.cu, solve.cu) and of the batch kernels
// (persistent.cu).
#pragma once

#include "internal.h"

#include <cuda_runtime.h>

// Threads per CTA of the whole-step launch (several Newton iterations) and of the team assembly; the
// single-Newton solve launch sets its own (kSolveMaxThreads).
#ifndef B3G_PCG_THREADS
#define B3G_PCG_THREADS 256
#endif

namespace b3g {

// Storage / arithmetic of the PCG: matrix storage type and vector type.
enum Prec
{
	kP32 = 0,   // float blocks, float vectors, double dot products
	kP64 = 1,   // double blocks and vectors
	kPBF = 2    // bf16 blocks in the iteration, float blocks for the residual refresh, float vectors
};

// What the row assembly sets up for the PCG besides pb and the Jacobi: nothing, r = pb, s = d =
// M^-1 r and the zero initial guess, or only s = M^-1 pb (the grid team's solve sets up its other
// vectors itself).
enum { kInitNone = 0, kInitAll = 1, kInitTeam = 2 };

struct StepParamsHost
{
	float h;
	int first_newton;
};

cudaError_t op_elements(const DevBody& B, const StepParamsHost& P, cudaStream_t st);
cudaError_t op_assemble(const DevBody& B, const StepParamsHost& P, int prec, int init, cudaStream_t st);
// filtered contacts: contact update and per-vertex constraints (B.filt) at the start of a step
cudaError_t op_contact_filter(const DevBody& B, float h, cudaStream_t st);
// One PCG solve by the grid team (solve.cuh) and, for newton >= 0, what follows it in Newton
// iteration `newton` of a step: the final update, or the new iterate and the step's end once the
// Newton loop is done.
struct SolveArgs
{
	double tol2, newton_tol2;
	int max_iter, refresh;
	float h;
	int newton;        // Newton iteration of a body step; -1: only solve, the solution stays in py
	int newton_max;    // Newton iterations the step may take
	int forces_left;   // another Newton iteration may follow this one
	int warm;          // start from the solution at hand (r = b - A x) instead of zero
	int smem;          // bytes of shared memory of a CTA (set by op_solve)
	int keep;          // 1/1024 of a CTA's slices whose matrix stays in L2 (set by op_solve)
	int polls;         // of a team's wait before it gives up, 0: the default
};
// The team's reduction memory starts cleared, and the scalars without a fault (op_assemble does both).
cudaError_t op_solve(const DevBody& B, const SolveArgs& P, int prec, cudaStream_t st);
// The BF16 mode's solve (flexible CG on the FP32 blocks around `inner` PCG iterations with the BF16
// blocks) and what follows it. W: the inner solve's vectors, 4-wide, where shared memory has no
// room for them.
struct FcgVecs
{
	float *z, *r, *d, *q;
};
cudaError_t op_solve_fcg(const DevBody& B, const FcgVecs& W, const SolveArgs& P, int inner, cudaStream_t st);
// dt <= 0: no solve, only contact bookkeeping and clearing (body.cpp:552-604)
cudaError_t op_nostep(const DevBody& B, cudaStream_t st);
// clear a float array on the device
cudaError_t op_fill_f32(float* p, size_t count, float value, cudaStream_t st);

// One body of a batched host transfer: its state arrays and its place in the flat host array.
struct XferBody
{
	float* x;
	float* v;
	float* fext;
	unsigned long long off;  // first float of the body in the flat array
	unsigned n3;             // 3 * vertices
	unsigned pad;
};
// fext of every body += src[off .. off + n3) (one launch for the whole batch)
cudaError_t op_batch_scatter_add(const XferBody* table, uint32_t count, uint32_t max_n3, const float* src,
                                 cudaStream_t st);
// dst_x / dst_v[off .. off + n3) = x / v of every body (either may be null)
cudaError_t op_batch_gather(const XferBody* table, uint32_t count, uint32_t max_n3, float* dst_x, float* dst_v,
                            cudaStream_t st);
// Closest triangle-fixture hit of `count` segments (6 floats each, device): keys[r] (device,
// count entries) is reduced to fraction bits << 32 | triangle, then decoded into hits (device).
cudaError_t op_ray_cast(const DevBody& B, int ntri, const float* segments, uint32_t count, unsigned long long* keys,
                        b3g_ray_hit* hits, cudaStream_t st);

// The same for up to kRayPick segments (host) in one launch. scratch: zero before the first call, left
// zero; hits may be page-locked host memory.
constexpr uint32_t kRayPick = 64;
struct RaySegments
{
	float s[kRayPick][6];
};
struct RayScratch
{
	unsigned long long key[kRayPick];
	unsigned arrived[kRayPick];
};
cudaError_t op_ray_pick(const DevBody& B, int ntri, const float* segments, uint32_t count, RayScratch* scratch,
                        b3g_ray_hit* hits, cudaStream_t st);

// Persistent batch kernel: every body listed in `big` (teams of `cluster` CTAs) and in `small`
// (one CTA each) steps `steps` times in one launch.
struct BatchArgs
{
	const DevBody* bodies;   // device array of all bodies of the batch
	const int* big;          // device array: indices of bodies stepped by whole clusters
	int nbig;
	const int* small;        // device array: indices of bodies stepped by single CTAs
	int nsmall;
	// The solve launch's teams: body k of the order (big, then small) is solved by a team of
	// kMaxTeamCtas >> t CTAs for the first t with k < tier_end[t]; teams are at most `cluster` wide.
	int tier_end[kTiers];
	unsigned* queue;         // device: kQueueCounters work counters, cleared by op_batch
	int steps;
	float h;
	int newton;
	int max_iter;
	double tol2;
	int refresh;
	double newton_tol2;
	int prec;
	int cluster;             // CTAs per cluster: 1, 2, 4 or 8
	int ctas;                // CTAs of the launch (multiple of cluster)
	unsigned long long* prof; // optional phase cycle counters (8 per CTA), null = off
	int part = 0;            // single-Newton steps: 0 every launch, 1 assembly only, 2 PCG only
	cudaEvent_t ev_rows = nullptr;  // if set, recorded between the element and the row launches
	// up to kFlatNewton iterations: the elements, then the rows, of all bodies in two flat launches before
	// the PCG launch. elem_off[k] / slice_off[k]: first element / row slice of bodies[k] in the
	// flat numbering (count + 1 entries each; elements of a body: tetrahedra, triangles, springs,
	// stretch/shear triangles, mouse springs). Null = the team launches do both, as for many
	// Newton iterations.
	const unsigned* elem_off = nullptr;
	const unsigned* slice_off = nullptr;
	unsigned nelem = 0;
	unsigned nslices = 0;
	int nbodies = 0;
	int tets_only = 0;       // every body has tetrahedra only and no contact spheres
	int filter = 0;          // filtered contacts: bodies with a filt buffer; their vertices follow
	                         // their elements in the flat element numbering
	// Split assembly (side stream set): bodies below the flat element offset elem_mid (slice
	// offset slice_mid) form group 1, the rest group 2; group 2's elements run on `side`,
	// forked and joined through ev_fork / ev_join, concurrently with group 1's rows. CTAs per SM
	// of the element and row launches (0: their defaults).
	cudaStream_t side = nullptr;
	cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
	// A second solve launch on `side` (0: none): clusters of `helper` CTAs on the SMs that the first one's
	// clusters leave free, taking the bodies of teams at most that wide from the same counters.
	int helper = 0;
	int polls = 0;           // of a solve team's wait before it gives up, 0: the default
	unsigned elem_mid = 0, slice_mid = 0;
	int split_elem_per_sm = 0, split_rows_per_sm = 0;
};
// Two kinds of solve teams: the first nbig bodies by teams of `cluster` CTAs, the rest by one CTA.
inline void two_tiers(BatchArgs* A, int cluster, int nbig, int count)
{
	for (int t = 0; t < kTiers; ++t) A->tier_end[t] = t == kTiers - 1 ? count : ((kMaxTeamCtas >> t) <= cluster ? nbig : 0);
}
// Newton iterations of a batched step that take launches of their own (elements, rows, solve), ms a step
// in one launch -> in launches of their own: 12 uneven blocks x 3 iterations 3.3 -> 1.4, 160 blocks 9.5 ->
// 4.6, 24 blocks and cloths 33.8 -> 11.8; 16 allowed and two or three taken 2.3 -> 1.3, 6.1 -> 3.8. An
// allowed iteration that no body takes costs its launches some 10 us, so a step that may take more is
// one launch of the whole-step kernel, which stops at each body's last iteration.
constexpr int kFlatNewton = 16;
cudaError_t op_batch(const BatchArgs& A, cudaStream_t st);
// Co-resident clusters of the batch kernel for this precision and cluster size (0 on error).
int batch_max_clusters(int prec, int cluster);

} // namespace b3g
