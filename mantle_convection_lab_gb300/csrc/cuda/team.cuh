// The team of blocks that runs one converged solve, shared by the uniform
// (k_mg.cu) and the refined-mesh (k_qt.cu) solvers: the whole cooperative
// grid (one model per launch), one thread-block cluster of a batched launch,
// or one block of a batched launch.
#pragma once
#include "mclg_dev.cuh"

namespace mclg {

// The blocks that share a pass over a level: block `rank` of `size` (the
// whole grid, a thread-block cluster, or one block alone).
constexpr int kTeamThreads = 512;   // most threads of a team's block

struct Part {
	int rank, size;
	// This thread's number in the blocks of the pass: warps are dealt to the
	// blocks in turn, so that a loop of few trips uses many SMs.
	__device__ int thread() const { return (((threadIdx.x >> 5) * size + rank) << 5) + (threadIdx.x & 31); }
};

// ---- where a solve runs ---------------------------------------------------------
// The team of blocks that solves one model:
//   SYNC_GRID     the whole cooperative grid (grid barriers, deterministic
//                 grid reductions through global memory);
//   SYNC_CLUSTER  one thread-block cluster of a batch (cluster barriers,
//                 reductions over the blocks' shared memory, read through
//                 distributed shared memory in rank order);
//   SYNC_BLOCK    one block of a batch (block barriers and reductions).
enum { SYNC_GRID = 0, SYNC_CLUSTER = 1, SYNC_BLOCK = 2 };

// Few words, so that a solve keeps it in registers: what lies on the stack misses
// L1 after every team barrier (whose acquire empties it), an L2 access each time.
struct Sync {
	int mode;
	double *partials;            // the reductions' partials: SYNC_GRID [2][kRedWidth][kMaxCoopBlocks] in global
	                             // memory, SYNC_CLUSTER this block's [2][kRedWidth] in shared memory
	int flip;                    // which of the two partial buffers the next reduction writes (see GridRed)
	int rank, size;              // this block in the team
	// tid and nth for loops over nodes and elements: warps are dealt to the blocks
	// in turn (Part::thread)
	static __device__ Sync of(int mode, double *partials, int rank, int size)
	{
		Sync s;
		s.mode = mode;
		s.partials = partials;
		s.flip = 0;
		s.rank = rank;
		s.size = size;
		return s;
	}
	__device__ int tid() const { return Part{rank, size}.thread(); }
	__device__ int nth() const { return size * (int)blockDim.x; }
	__device__ void sync()
	{
		if (mode == SYNC_GRID)
			cg::this_grid().sync();
		else if (mode == SYNC_CLUSTER)
			cg::this_cluster().sync();
		else
			__syncthreads();
	}
	// Sums of NV values over the team, formed by warp 0 of every block from the
	// same partials in the same order; f(sums) runs on thread 0 of each block, and
	// what it writes to shared memory is visible to the block on return.  Each
	// value's thread partials go through shared memory to one warp (8 or 16, then 5
	// additions; blocks of 256 or 512 threads): a butterfly in every warp takes eight times that of the FP64
	// pipe, which has 2 lanes per clock and SM.
	__device__ static double *scratch()
	{
		__shared__ double sh[kRedWidth * kTeamThreads];
		return sh;
	}
	template <int NV, class F>
	__device__ __forceinline__ void reduce_then(const double (&v)[NV], F f)
	{
		static_assert(NV <= kRedWidth, "partials per reduction");
		double *sh = scratch();
		const int lane = threadIdx.x & 31;
#pragma unroll
		for (int k = 0; k < NV; k++)
			sh[k * kTeamThreads + threadIdx.x] = v[k];
		__syncthreads();
		double t[NV];
#pragma unroll
		for (int k = 0; k < NV; k++)
			t[k] = 0.0;
		if (threadIdx.x < 32) {
#pragma unroll
			for (int k = 0; k < NV; k++) {
				const double *s = sh + k * kTeamThreads + lane;
				t[k] = ((s[0] + s[32]) + (s[64] + s[96])) + ((s[128] + s[160]) + (s[192] + s[224]));
				if (blockDim.x > 256) {
					s += 256;
					t[k] += ((s[0] + s[32]) + (s[64] + s[96])) + ((s[128] + s[160]) + (s[192] + s[224]));
				}
				t[k] = warp_sum(t[k]);
			}
		}
		if (mode == SYNC_GRID) {
			double *buf = partials + (size_t)flip * kMaxCoopBlocks * kRedWidth;
			if (threadIdx.x == 0) {
#pragma unroll
				for (int k = 0; k < NV; k++)
					buf[k * kMaxCoopBlocks + rank] = t[k];
			}
			cg::this_grid().sync();
			if (threadIdx.x < 32) {
#pragma unroll
				for (int k = 0; k < NV; k++) {
					double a0 = 0.0, a1 = 0.0;
					int b = lane;
					for (; b + 32 < size; b += 64) {
						a0 += buf[k * kMaxCoopBlocks + b];
						a1 += buf[k * kMaxCoopBlocks + b + 32];
					}
					if (b < size)
						a0 += buf[k * kMaxCoopBlocks + b];
					t[k] = warp_sum(a0 + a1);
				}
			}
			flip ^= 1;
		} else if (mode == SYNC_CLUSTER) {
			double *mine = partials + flip * kRedWidth;
			if (threadIdx.x == 0) {
#pragma unroll
				for (int k = 0; k < NV; k++)
					mine[k] = t[k];
			}
			cg::cluster_group cl = cg::this_cluster();
			cl.sync();
			if (threadIdx.x < 32) {
				const double *other = cl.map_shared_rank(mine, lane < size ? lane : 0);
#pragma unroll
				for (int k = 0; k < NV; k++)
					t[k] = warp_sum(lane < size ? other[k] : 0.0);
			}
			flip ^= 1;
		}
		if (threadIdx.x == 0)
			f(t);
		__syncthreads();
	}
	// The sums in every thread.
	template <int NV>
	__device__ __forceinline__ void reduce(double (&v)[NV])
	{
		__shared__ double out[NV];
		reduce_then<NV>(v, [&](const double (&t)[NV]) {
#pragma unroll
			for (int k = 0; k < NV; k++)
				out[k] = t[k];
		});
#pragma unroll
		for (int k = 0; k < NV; k++)
			v[k] = out[k];
	}
	__device__ bool leader() const { return rank == 0; }
	// the blocks of a pass: the team for team-wide levels, this block alone otherwise
	__device__ Part part(bool wide) const { return wide ? Part{rank, size} : Part{0, 1}; }
	__device__ void sync(bool wide)
	{
		if (wide)
			sync();
		else
			__syncthreads();
	}
};

// A solver's arguments copied to shared memory: functions take references into
// them, which for kernel parameters would copy them to every thread's stack and
// for a batch's arguments would read global memory after every barrier.
template <class A>
__device__ void load_args(A &to, const A &from)
{
	static_assert(sizeof(A) % 4 == 0, "copied by words");
	const unsigned *s = reinterpret_cast<const unsigned *>(&from);
	unsigned *d = reinterpret_cast<unsigned *>(&to);
	for (int i = threadIdx.x; i < (int)(sizeof(A) / 4); i += blockDim.x)
		d[i] = s[i];
	__syncthreads();
}

}  // namespace mclg
