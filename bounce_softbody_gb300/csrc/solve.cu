// Launch of the grid team's PCG (solve.cuh).
#include "solve.cuh"
#include "solve_rule.h"

#include <algorithm>
#include <cstdlib>

namespace b3g {

namespace {

struct Device
{
	int sms = 1, room = 0;  // SMs a team may use, dynamic shared memory of a CTA
};

const Device& device()
{
	static const Device d = [] {
		Device v;
		int dev = 0;
		cudaGetDevice(&dev);
		cudaDeviceGetAttribute(&v.sms, cudaDevAttrMultiProcessorCount, dev);
		int smem = 0;
		cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
		v.room = (smem - (int)sizeof(SolveSh) - 128) & ~127;
		v.sms = std::max(1, std::min(v.sms, kTeamMax));
		return v;
	}();
	return d;
}

// A CTA takes consecutive slices, one warp each up to 16 warps (128 registers a thread; 1024 threads
// at 64 registers spill in the sweep: 64^3 block 13.6 ms a step against 11.1). At least four slices a
// CTA: on small bodies fewer CTAs make the sums cheaper than more CTAs make the sweeps (10^3 block,
// 32 slices: 32 / 16 / 8 / 4 CTAs 263 / 265 / 256 / 300 us a step).
// keep: what shared memory does not hold of the matrix goes through L2 once per iteration. Up to
// kL2Keep bytes of it all stay there. Beyond, a cyclic sweep under LRU would find nothing left, so
// kL2Keep bytes are kept (evict last) and the rest streams past them (evict first). 64^3 block,
// 165 MB: 0 / 25 / 37 / 50 / 62 / 75 / 100 % kept 12.8 / 12.4 / 12.0 / 11.7 / 12.7 / 13.6 / 14.1 ms.
// Row vectors that shared memory does not hold are read and written every iteration, so their bytes come
// off kL2Keep first: matrix kept beside them pushed them out. BF16 62^3 3.51 -> 3.15 ms a step, 75x74x73
// 6.08 -> 5.45, 97x89x83 10.9 -> 9.3 (10.2 kernel by kernel); FP32 97x89x83 11.1 -> 10.5 ms per 100 iterations,
// 62^3, whose vectors fit, the same.
constexpr size_t kL2Keep = (size_t)80 << 20;

struct Geometry
{
	int ctas, threads, smem, keep;
};

Geometry geometry(const DevBody& B, size_t vec_bytes, size_t slot_bytes, int least)
{
	const Device& dv = device();
	const int per = std::max(least, (B.nslices + dv.sms - 1) / dv.sms);
	Geometry g;
	g.ctas = std::max(1, (B.nslices + per - 1) / per);
	const int slices = (B.nslices + g.ctas - 1) / g.ctas;
	const int rounds = (slices + kSolveMaxThreads / 32 - 1) / (kSolveMaxThreads / 32);
	g.threads = 32 * std::max(1, (slices + rounds - 1) / rounds);
	const size_t want = (size_t)slices * (vec_bytes + (size_t)B.maxw * kSlice * slot_bytes);
	const size_t room = (size_t)(g.threads <= 256 ? dv.room : dv.room - kL1Room);
	g.smem = (int)(std::min(want, room) & ~(size_t)127);
	const size_t total = (size_t)B.nslots * slot_bytes;
	const size_t held = (size_t)g.ctas * (size_t)std::max(0, g.smem - (int)std::min<size_t>(slices * vec_bytes, g.smem));
	const size_t stream = total > held ? total - held : 0;
	const size_t outside = (size_t)g.ctas * (slices * vec_bytes - std::min<size_t>(slices * vec_bytes, g.smem));
	const size_t keep = kL2Keep > outside ? kL2Keep - outside : 0;
	g.keep = stream <= keep ? 1024 : (int)(1024 * keep / stream);
	return g;
}

// A cooperative launch: the CTAs of the team wait for one another, so all have to be resident.
template <class... Args>
cudaError_t launch_team(void (*kernel)(Args...), const Geometry& g, cudaStream_t st, Args... args)
{
	cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, device().room);
	if (e != cudaSuccess) return e;
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3((unsigned)g.ctas, 1, 1);
	cfg.blockDim = dim3((unsigned)g.threads, 1, 1);
	cfg.dynamicSmemBytes = (size_t)g.smem;
	cfg.stream = st;
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeCooperative;
	attr[0].val.cooperative = 1;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// The launch of one cluster of `cl` CTAs
template <class... Args>
cudaError_t cluster_config(void (*kernel)(Args...), int cl, int threads, int smem, cudaStream_t st, cudaLaunchConfig_t* cfg,
                           cudaLaunchAttribute* attr)
{
	cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, device().room);
	if (e == cudaSuccess && cl > 8) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
	*cfg = {};
	cfg->gridDim = dim3((unsigned)cl, 1, 1);
	cfg->blockDim = dim3((unsigned)threads, 1, 1);
	cfg->dynamicSmemBytes = (size_t)smem;
	cfg->stream = st;
	attr->id = cudaLaunchAttributeClusterDimension;
	attr->val.clusterDim.x = (unsigned)cl;
	attr->val.clusterDim.y = 1;
	attr->val.clusterDim.z = 1;
	cfg->attrs = attr;
	cfg->numAttrs = 1;
	return e;
}

// The widest cluster that the device can hold, 0 if none: 16 CTAs need a GPC with as many SMs for them,
// which a part of a device need not have. B3G_SOLVE_CLUSTER caps it (read once).
template <class... Args>
int widest_cluster(void (*kernel)(Args...))
{
	const char* cap = std::getenv("B3G_SOLVE_CLUSTER");
	for (int cl = kMaxTeamCtas; cl > 0; cl /= 2)
	{
		cudaLaunchConfig_t cfg;
		cudaLaunchAttribute attr;
		int clusters = 0;
		if (!(cap && cl > std::atoi(cap)) && cluster_config(kernel, cl, 256, device().room, nullptr, &cfg, &attr) == cudaSuccess &&
		    cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0)
			return cl;
		cudaGetLastError();
	}
	return 0;
}

template <class TA, class TV, bool FF, bool FILTER>
cudaError_t launch_cluster(const DevBody& B, SolveArgs P, int cl, cudaStream_t st)
{
	auto* kernel = k_solve_cluster<TA, TV, FF, FILTER>;
	const int slices = (B.nslices + cl - 1) / cl;
	const size_t want = (size_t)slices * (solve_vec_bytes<TV, FF>() + (size_t)B.maxw * kSlice * solve_slot_bytes<TA>());
	P.smem = (int)(std::min(want, (size_t)device().room) & ~(size_t)127);
	P.keep = 1024;
	cudaLaunchConfig_t cfg;
	cudaLaunchAttribute attr;
	cudaError_t e = cluster_config(kernel, cl, 32 * slices, P.smem, st, &cfg, &attr);
	return e == cudaSuccess ? cudaLaunchKernelEx(&cfg, kernel, B, P) : e;
}

template <class TA, class TV, bool FF, bool FILTER>
cudaError_t launch_solve(const DevBody& B, SolveArgs P, cudaStream_t st)
{
	static const int widest = widest_cluster(k_solve_cluster<TA, TV, FF, FILTER>);
	const int cl = cluster_ctas(B.nslices, widest);
	if (cl > 0) return launch_cluster<TA, TV, FF, FILTER>(B, P, cl, st);
	// FP64 sweeps wait for the FP64 pipe, so they spread over every SM
	const Geometry g = geometry(B, solve_vec_bytes<TV, FF>(), solve_slot_bytes<TA>(), sizeof(TV) == 8 ? 1 : 4);
	P.smem = g.smem;
	P.keep = g.keep;
	if (g.threads <= 256) return launch_team(k_solve<TA, TV, FF, FILTER, 256>, g, st, B, P);
	return launch_team(k_solve<TA, TV, FF, FILTER, 512>, g, st, B, P);
}

template <bool FILTER>
cudaError_t launch_fcg(const DevBody& B, const FcgVecs& W, SolveArgs P, int inner, cudaStream_t st)
{
	const Geometry g = geometry(B, kFcgVecBytes, solve_slot_bytes<__nv_bfloat16>(), 4);
	P.smem = g.smem;
	P.keep = g.keep;
	if (g.threads <= 256) return launch_team(k_solve_fcg<FILTER, 256>, g, st, B, W, P, inner);
	return launch_team(k_solve_fcg<FILTER, 512>, g, st, B, W, P, inner);
}

} // namespace

cudaError_t op_solve(const DevBody& B, const SolveArgs& P, int prec, cudaStream_t st)
{
	if (prec == kP64)
		return B.filt ? launch_solve<double, double, false, true>(B, P, st) : launch_solve<double, double, false, false>(B, P, st);
	if (!B.xff) return launch_solve<float, float, false, false>(B, P, st);
	return B.filt ? launch_solve<float, float, true, true>(B, P, st) : launch_solve<float, float, true, false>(B, P, st);
}

cudaError_t op_solve_fcg(const DevBody& B, const FcgVecs& W, const SolveArgs& P, int inner, cudaStream_t st)
{
	return B.filt ? launch_fcg<true>(B, W, P, inner, st) : launch_fcg<false>(B, W, P, inner, st);
}

} // namespace b3g
