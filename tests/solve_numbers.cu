// Team sums of the solve launches on given values, the grid's and a cluster's, fenced and not, and their
// divisions.
#include "solve.cuh"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

using namespace b3g;

namespace numbers {

constexpr int kWarpsMax = 16, kRounds = 24;

// value r of warp w of CTA c at ((c * warps) + w) * kRounds + r; CTA c's total at c * kRounds + r
template <class T>
__device__ void sums(T& team, const double* in, double* out)
{
	const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5;
	for (int r = 0; r < kRounds; ++r)
	{
		const Fixed v = to_fixed(in[((size_t)blockIdx.x * warps + warp) * kRounds + r]);
		const double t = r % 3 == 2 ? team.template sum<true>(v) : team.template sum<false>(v);
		if (threadIdx.x == 0) out[(size_t)blockIdx.x * kRounds + r] = team.ok ? t : -1.0;
	}
}

__global__ void grid_sums(const double* in, double* out, TeamMemory* mem)
{
	__shared__ SolveSh sh;
	GridTeam<double> team(&sh, mem, 0);
	sums(team, in, out);
}

__global__ void cluster_sums(const double* in, double* out)
{
	__shared__ SolveSh sh;
	ClusterTeam<double> team(&sh, 0);
	cooperative_groups::this_cluster().sync();
	team.form((int)cooperative_groups::this_cluster().num_blocks());
	sums(team, in, out);
	cooperative_groups::this_cluster().sync();
}

__global__ void divisions(const double* in, double* out, int count)
{
	const int k = blockIdx.x * blockDim.x + threadIdx.x;
	if (k < count) out[k] = (double)Divisor<float>(in[2 * k + 1]).divide(in[2 * k]);
}

bool ok(cudaError_t e)
{
	if (e != cudaSuccess) std::fprintf(stderr, "%s\n", cudaGetErrorString(e));
	return e == cudaSuccess;
}

} // namespace numbers

// stdin: ctas, warps, cluster (0: the grid), then ctas * warps * kRounds doubles; stdout: ctas * kRounds.
// Or: count, 0, -1, then count pairs of doubles; stdout: count quotients.
int main()
{
	using namespace numbers;
	int shape[3];
	while (std::fread(shape, sizeof(int), 3, stdin) == 3)
	{
		const int ctas = shape[0], warps = shape[1], cluster = shape[2];
		if (cluster < 0)
		{
			const int count = ctas;
			if (count < 1 || count > 1 << 24) return 2;
			std::vector<double> in(2 * (size_t)count), out(count);
			if (std::fread(in.data(), sizeof(double), in.size(), stdin) != in.size()) return 2;
			double *din = nullptr, *dout = nullptr;
			if (!ok(cudaMalloc(&din, in.size() * sizeof(double))) || !ok(cudaMalloc(&dout, out.size() * sizeof(double))) ||
			    !ok(cudaMemcpy(din, in.data(), in.size() * sizeof(double), cudaMemcpyHostToDevice)))
				return 3;
			divisions<<<(count + 255) / 256, 256>>>(din, dout, count);
			if (!ok(cudaGetLastError()) || !ok(cudaMemcpy(out.data(), dout, out.size() * sizeof(double), cudaMemcpyDeviceToHost))) return 3;
			cudaFree(din);
			cudaFree(dout);
			std::fwrite(out.data(), sizeof(double), out.size(), stdout);
			continue;
		}
		if (ctas < 1 || ctas > kTeamMax || warps < 1 || warps > kWarpsMax || (cluster && cluster != ctas) || cluster > kMaxTeamCtas) return 2;
		std::vector<double> in((size_t)ctas * warps * kRounds), out((size_t)ctas * kRounds);
		if (std::fread(in.data(), sizeof(double), in.size(), stdin) != in.size()) return 2;
		double *din = nullptr, *dout = nullptr;
		TeamMemory* mem = nullptr;
		if (!ok(cudaMalloc(&din, in.size() * sizeof(double))) || !ok(cudaMalloc(&dout, out.size() * sizeof(double))) ||
		    !ok(cudaMalloc(&mem, sizeof(TeamMemory))) || !ok(cudaMemset(mem, 0, sizeof(TeamMemory))) ||
		    !ok(cudaMemcpy(din, in.data(), in.size() * sizeof(double), cudaMemcpyHostToDevice)))
			return 3;
		cudaLaunchConfig_t cfg = {};
		cfg.gridDim = dim3((unsigned)ctas);
		cfg.blockDim = dim3((unsigned)(32 * warps));
		cudaLaunchAttribute attr = {};
		cfg.attrs = &attr;
		cfg.numAttrs = 1;
		cudaError_t e = cudaSuccess;
		if (cluster)
		{
			attr.id = cudaLaunchAttributeClusterDimension;
			attr.val.clusterDim.x = (unsigned)cluster;
			attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
			if (cluster > 8) e = cudaFuncSetAttribute(cluster_sums, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
			if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, cluster_sums, (const double*)din, dout);
		}
		else
		{
			attr.id = cudaLaunchAttributeCooperative;
			attr.val.cooperative = 1;
			e = cudaLaunchKernelEx(&cfg, grid_sums, (const double*)din, dout, mem);
		}
		if (!ok(e) || !ok(cudaDeviceSynchronize()) ||
		    !ok(cudaMemcpy(out.data(), dout, out.size() * sizeof(double), cudaMemcpyDeviceToHost)))
			return 3;
		cudaFree(din);
		cudaFree(dout);
		cudaFree(mem);
		std::fwrite(out.data(), sizeof(double), out.size(), stdout);
	}
	return 0;
}
