// The fused substep.
#pragma once
#include "tiles.cuh"

namespace xpbd {
namespace dev {

// ===========================================================================
// The whole substep in one cooperative launch: predict, then per iteration distance,
// volume solve and gather, shape matching and the projections, then the velocity
// commit, with a grid-wide barrier between phases.  Every phase runs the same
// per-item code as its own kernel (the *_row / *_lane / tile functions, with plain
// loads for the data the launch itself writes), so the result is that of the kernel
// sequence to FP32 rounding; what changes is one launch per substep instead of one per
// phase.  Covers the default forms (Jacobi distance, 4-lane one-pass volume solve and
// gather, shape matching, colliders, ground, press, contact shapes); self-collision,
// object mode and the Gauss-Seidel forms keep the kernel sequence.
// ===========================================================================
struct SubstepArgs {
	int n, iters, use_distance, use_volume, use_shape, shape_robust, project;
	const StepParams* P;
	float4 *pos_curr, *pos_next, *pos_tmp, *vel;
	float* lam_vol;
	const float4* cshape;
	const float* crmax;
	float* crg;
	const int *off, *nbr;
	const float *ndist, *nstiff;
	float* lam;
	const int *vol_off, *vol_group, *mat_type, *rev_off, *rev_idx;
	const int4* vol_pack;
	const VolTile* tiles;
	const int* tile_rows;
	const unsigned int* tile_words;
	int tile_count, list_count;
	const int* list_rows;
	const float *det_rest, *rest_len;
	float4* rec;
	float* recz;
	const float4 *pos_rest, *shape_rest;
	float4* shape_q;
	DevCounters* ctr;
	const int* obj_id;
	const KinCollider* ext_kin;
	const int2* ext_range;
	float* pos_out3;
	const int* perm;
};

// Grid-wide barrier of the fused launch (all blocks are co-resident: the launch is
// cooperative).  Thread 0 of each block publishes its block's writes, arrives, and the
// last to arrive opens the next generation; the wait is bounded (about 2^24 polls of at
// least 64 ns): if it runs out, bar_timeout is set and the launch runs to its end with
// the host reporting the error, instead of hanging the GPU.
__device__ __forceinline__ void grid_barrier(DevCounters* __restrict__ ctr)
{
	__syncthreads();
	if (threadIdx.x == 0) {
		volatile unsigned int* gen = &ctr->bar_gen;
		const unsigned int g = *gen;
		__threadfence();
		if (atomicAdd(&ctr->bar_count, 1u) + 1u == gridDim.x) {
			ctr->bar_count = 0u;
			__threadfence();
			atomicAdd(&ctr->bar_gen, 1u);
		}
		else {
			unsigned int polls = 0;
			while (*gen == g) {
				if (++polls > (1u << 24)) { atomicExch(&ctr->bar_timeout, 1u); break; }
				__nanosleep(64);
			}
		}
		__threadfence();
	}
	__syncthreads();
}

__global__ void __launch_bounds__(kBlock, 2) k_substep_fused(SubstepArgs A)
{
	extern __shared__ __align__(16) unsigned char slab[];   // kVtSmem
	__shared__ unsigned int part[2][kVtThreads / 32];
	__shared__ SolveSums sums[kBlock / 32];
	DevCounters* ctr = A.ctr;
	const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	const long long nth = (long long)gridDim.x * blockDim.x;
	const int lane = threadIdx.x & 31;
	const long long wbase = tid - lane;   // lane-group phases: whole warps iterate together
	const int n = A.n;
	const StepParams* P = A.P;
	for (long long i = tid; i < n; i += nth)
		predict_row((int)i, n, P, A.pos_curr, A.pos_next, A.vel, A.use_volume ? A.lam_vol : nullptr, A.cshape, A.crg);
	grid_barrier(ctr);
	float4* pin = A.pos_next;
	float4* pout = A.pos_tmp;
	for (int it = 0; it < A.iters; ++it) {
		const int first = (it == 0), last = (it == A.iters - 1);
		if (A.use_distance) {
			for (long long i = tid; i < n; i += nth)
				distance_row<false>((int)i, n, P, pin, pout, A.off, A.nbr, A.ndist, A.nstiff, A.lam, first ? 0 : 1,
					last ? 0 : 1);
			grid_barrier(ctr);
			float4* t = pin; pin = pout; pout = t;
		}
		if (A.use_volume) {
			for (long long b = wbase; b < n; b += nth) {
				solve_warp<4, false>(sums[threadIdx.x >> 5], (int)b, n, P, pin, A.vol_off, A.vol_group, A.vol_pack, A.det_rest, A.mat_type,
					A.lam_vol, A.rec, A.recz, first ? 0 : 1);
				__syncwarp();
			}
			grid_barrier(ctr);
			for (int t = blockIdx.x; t < A.tile_count; t += gridDim.x) {
				tile_gather<false>(slab, part, n, P, pin, pout, A.tiles + t, A.tile_rows, A.tile_words, A.rev_off, A.rev_idx,
					A.rec, A.recz, A.rest_len);
				__syncthreads();
			}
			for (long long b = wbase; b < 4LL * A.list_count; b += nth)
				gather_group_lane<4>((long long)ordered_node(A.list_rows, (int)(b + lane) / 4, A.list_count, n) * 4 +
					(lane & 3), n, P, pin, pout, A.rev_off, A.rev_idx, A.rec, A.recz, A.rest_len);
			grid_barrier(ctr);
			float4* t = pin; pin = pout; pout = t;
		}
		if (A.use_shape) {
			for (long long i = tid; i < n; i += nth) {
				auto at = [&](int e) { return __ldg(A.nbr + e); };
				if (A.shape_robust)
					shape_row<true, false>((int)i, n, P, pin, pout, A.pos_rest, A.off, at, A.shape_rest, A.shape_q);
				else
					shape_row<false, false>((int)i, n, P, pin, pout, A.pos_rest, A.off, at, A.shape_rest, A.shape_q);
			}
			grid_barrier(ctr);
			float4* t = pin; pin = pout; pout = t;
		}
		if (A.project) {
			for (long long i = tid; i < n; i += nth)
				project_row((int)i, n, P, pin, A.pos_curr, nullptr, nullptr, A.ctr, last ? 1 : 0, A.obj_id, A.ext_kin,
					A.ext_range, nullptr, nullptr, A.cshape, A.crmax, A.crg);
			grid_barrier(ctr);
		}
	}
	for (long long i = tid; i < n; i += nth) velocity_row((int)i, n, P, A.pos_curr, pin, A.vel, A.pos_out3, A.perm, A.crg);
}

}  // namespace dev
}  // namespace xpbd
