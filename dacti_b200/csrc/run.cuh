// A run of ACTI-level substeps in one launch: the scheduler of Integrator::integrate
// (impl/integrate.hpp:25-67) and every stage of a substep in one persistent kernel, with a barrier over
// the launch's blocks between stages that depend on one another.
//
// What bounds a substep of a small cluster is not its cells but its chain of launches: a substep is about
// twenty stage kernels and one host synchronisation, 100 to 200 us on this GPU whatever the cluster's
// size, while the stages' own work on a few thousand cells is a microsecond or two each. Here a barrier
// takes the place of a launch, stages that do not read one another's results share one (six to nine
// barriers a substep), and the host is not asked until the global step ends or something needs it. A step with a
// substep callback, with stage timing or with other stage options takes the launches.
#pragma once

#include "stages.cuh"

namespace dg {

// Schedule state of one solver (Integrator: max_acti_level, acti_counter, acti_time, and this port's stamp
// and epoch counters), kept on the device while a run executes.
struct TreeSched {
	int max_acti, stamp, epoch, pad;
	int counter[MAX_ACTI];
	double time[MAX_ACTI];
};

// Epochs of one substep (Solver::substep): update + 1, slope + 2, the four multiphase sweeps + 3 .. + 6,
// then the estimate, the split and the unsplit.
template<class M>
constexpr int EPOCH_EST = M::MULTI ? 7 : 3;
template<class M>
constexpr int SUBSTEP_EPOCHS = EPOCH_EST<M> + 2;

// Why a run returned. The cursor (seq, l) stands after the last substep that was begun.
enum RunStop : int {
	RUN_DONE = 0,   // the global step is complete
	RUN_STATUS,     // the last substep left a status (a NaN or an error)
	RUN_LARGE,      // the next cluster is outside the run's range; nothing of its substep has run
	RUN_CAPACITY,   // the split requests of substep `L` do not fit the pool; its head has run, its tail has not
};

struct RunState {
	TreeSched sch;
	int seq, l;  // sequence value, and the next level index to look at in it (MAX_ACTI: the next value is due)
	int stop, L;
	long long splits, unsplits, updates, substeps;
	int32_t *clu[MAX_ACTI], *tmp;  // the list pointers as the run left them
};

struct RunArgs {
	Pool P;
	Consts C;
	BcTable B;
	Lists Ls;
	Counters *cnt;
	RunState in;
	RunState *out;      // host memory: the state as the run left it, written last
	Counters *out_cnt;  // host memory: the counters
	unsigned *bar;    // grid barrier: arrivals since the launch
	double global_dt;
	int limiter, sigma;
	int rows;         // largest cluster the run takes
	int clustered;    // the launch is one thread-block cluster: its hardware barrier is the run's
};

constexpr int RUN_THREADS = 512;

// The warp items of a run: dealt out over the blocks one by one, so that few items spread over all SMs and the
// cells with long walks (hanging faces, subtree means), which lie side by side in the list, do not meet in one
// block: the slowest block ends a stage (2 to 3% on clusters below ten thousand cells against contiguous chunks). `rev` hands
// the items to the blocks' warps from the last one on, for the second of two stages that share a barrier: with
// few items the two then run on different warps instead of one after the other.
struct DealtGrid {
	static constexpr bool DEEP = true, EARLY = true;
	int block, blocks;
	bool rev;
	__device__ __forceinline__ int begin(int) const {
		const int w = threadIdx.x >> 5;
		return (rev ? RUN_THREADS / 32 - 1 - w : w) * blocks + block;
	}
	__device__ __forceinline__ int end(int items) const { return items; }
	__device__ __forceinline__ int step() const { return blocks * (RUN_THREADS / 32); }
};

// A wait longer than this many polls (seconds of them) gives up: the launch ends without leaving a state, and the host
// takes the solver for lost. All blocks of a run are on the GPU together, so a wait is as long as the slowest block's
// stage, microseconds to milliseconds; polls, unlike a clock, stand still where another process has the GPU.
constexpr int BARRIER_POLLS = 1 << 23;

// Every thread of the launch arrives and leaves; writes before it are visible after it. False when the
// wait gave up, on every thread of the block.
__device__ __forceinline__ bool run_barrier(const RunArgs &a, unsigned &arrivals, int *s_ok) {
	if (a.clustered) {
		__syncthreads();
		asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
		return true;
	}
	arrivals += gridDim.x;
	__syncthreads();
	if (threadIdx.x == 0) {
		unsigned seen;
		asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(seen) : "l"(a.bar) : "memory");
		int polls = 0;
		++seen;
		while ((int) (seen - arrivals) < 0 && ++polls < BARRIER_POLLS)
			asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.bar) : "memory");
		*s_ok = (int) (seen - arrivals) >= 0;
	}
	__syncthreads();
	return *s_ok;
}

// The cluster's reassignment for a run: the cells that stay are listed chunk by chunk in their list order
// (a contiguous chunk per block, one reservation per block of RUN_THREADS cells), so that neighbours in the list stay neighbours.
template<class M>
__device__ __forceinline__ void run_reassign(const DealtGrid &g, const Pool &P, const Consts &C, const int32_t *list, int n, int L,
                                             double dtL, int counter_L, const Lists &Ls, Counters *cnt, int *s_warp /*[33]*/) {
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = RUN_THREADS / 32;
	const int items = warp_items(n, 32);
	const int first = (int) ((long long) items * g.block / g.blocks), last = (int) ((long long) items * (g.block + 1) / g.blocks);
	for (int base = first; base < last; base += nw) {
		const int tid  = (base + w) * 32 + lane;
		const bool in  = base + w < last && tid < n;
		const int i    = in ? list[tid] : 0;
		const bool st  = in && reassign_cell<M>(P, C, i, L, dtL, counter_L, Ls, cnt);
		const unsigned m = __ballot_sync(0xffffffffu, st);
		if (lane == 0) s_warp[w] = __popc(m);
		__syncthreads();
		if (w == 0) {
			const int v = lane < nw ? s_warp[lane] : 0;
			int x       = v;
#pragma unroll
			for (int o = 1; o < 32; o <<= 1) {
				const int y = __shfl_up_sync(0xffffffffu, x, o);
				if (lane >= o) x += y;
			}
			const int total = __shfl_sync(0xffffffffu, x, 31);
			int at          = 0;
			if (lane == 0 && total > 0) at = atomicAdd(&cnt->n_tmp, total);
			at = __shfl_sync(0xffffffffu, at, 0);
			if (lane < nw) s_warp[lane] = at + x - v;
		}
		__syncthreads();
		if (st) {
			const int at = s_warp[w] + __popc(m & ((1u << lane) - 1u));
			if (at < P.cap) Ls.tmp[at] = i;
			else set_status(&cnt->status, ST_CAPACITY);
		}
		__syncthreads();
	}
}

template<class M, bool V, class S>
__global__ void __launch_bounds__(RUN_THREADS, 1) k_run(const __grid_constant__ RunArgs a) {
	constexpr int NC = 1 << M::D, EX = EPOCH_EST<M>;
	__shared__ Lists s_ls;
	__shared__ TreeSched s;
	__shared__ int s_clu[MAX_ACTI];
	__shared__ int s_warp[33];
	__shared__ int s_seq, s_l, s_L, s_n, s_top, s_stop, s_ok;
	__shared__ long long s_tot[4];
	const Pool &P   = a.P;
	const Consts &C = a.C;
	Counters *cnt   = a.cnt;
	const int top_seq = 1 << (MAX_ACTI - 1);
	unsigned arrivals = 0;
	const bool lead   = threadIdx.x == 0;
	const DealtGrid g{(int) blockIdx.x, (int) gridDim.x, false}, r{(int) blockIdx.x, (int) gridDim.x, true};

	if (lead) {
		s     = a.in.sch;
		s_seq = a.in.seq;
		s_l   = a.in.l;
		s_ls  = a.Ls;
		s_top = cnt->top;
		for (int l = 0; l < MAX_ACTI; ++l) s_clu[l] = cnt->clu[l];
		s_tot[0] = s_tot[1] = s_tot[2] = s_tot[3] = 0;
		s_stop = -1;
	}
	if (lead && blockIdx.x == 0) {
		cnt->n_recv = cnt->n_defer = cnt->n_split = cnt->n_unsplit = cnt->n_new = cnt->n_tmp = 0;
		cnt->status = cnt->face_status = 0;
	}
	// every block has read the counters before any changes them
	if (!run_barrier(a, arrivals, &s_ok)) return;
	while (true) {
		// the next substep, on every block alike (impl/integrate.hpp:25-39)
		if (lead && s_stop < 0) {
			s_L = -1;
			while (s_L < 0) {
				if (s_l >= MAX_ACTI) {
					int finest = s.max_acti;
					for (int l = MAX_ACTI - 1; l > finest; --l)
						if (s_clu[l] > 0) {
							finest = l;
							break;
						}
					const int stride = 1 << (MAX_ACTI - 1 - finest);
					s_seq            = (s_seq / stride + 1) * stride;
					s_l              = 0;
					if (s_seq > top_seq) {
						s_stop = RUN_DONE;
						break;
					}
				}
				for (; s_l < MAX_ACTI && s_L < 0; ++s_l) {
					if (s_seq & ((1 << s_l) - 1)) continue;
					const int L = MAX_ACTI - s_l - 1;
					if (s_clu[L] > 0 && L > s.max_acti) {
						s.max_acti = L;
						s.time[L]  = s.time[L - 1];
					}
					if (L > s.max_acti) continue;
					s_L = L;
				}
			}
			if (s_L >= 0) {
				s_n = s_clu[s_L];
				if (s_n > a.rows) {
					s_stop = RUN_LARGE;
					--s_l;  // the level is due again
				} else {
					++s.stamp;
				}
			}
		}
		__syncthreads();
		if (s_stop >= 0) break;
		const int L = s_L, n = s_n, counter_L = s.counter[L], epoch0 = s.epoch, stamp = s.stamp;
		const double dtL    = a.global_dt / (double) (1 << L);
		const int32_t *list = s_ls.clu[L];
		const int e_upd     = epoch0 + 1;

		// the list of new cells, not in use before the regrid, holds the deferred cells' positions
		// `status` decides at a substep's end whether the run stops, and a block that is ahead may be here before the
		// others have read it: the face sums have a word of their own
		d_face_sum<M, V, S>(g, P, C, a.B, list, n, L, dtL, stamp, s_ls.recv, s_ls.fresh, cnt, &cnt->face_status);
		d_stamp(r, P, list, n, e_upd, cnt);
		if (!run_barrier(a, arrivals, &s_ok)) return;
		if (lead && blockIdx.x == 0) atomicOr(&cnt->status, __ldcg(&cnt->face_status));
		// the receivers are cells of slower clusters, the updated cells those of this one
		const bool deferred = __ldcg(&cnt->n_defer) > 0;
		if (deferred) d_deferred<M, S>(g, P, list, s_ls.fresh, &cnt->n_defer, L, cnt);
		if (__ldcg(&cnt->n_recv) > 0) d_flux_receive<M, S>(r, P, s_ls.recv, &cnt->n_recv, L, cnt);
		if (deferred && !run_barrier(a, arrivals, &s_ok)) return;
		d_update<M, V>(g, P, C, list, n, dtL, cnt);
		if (lead && blockIdx.x == 0) cnt->n_split = cnt->n_unsplit = cnt->n_new = cnt->n_tmp = 0;
		if (!run_barrier(a, arrivals, &s_ok)) return;
		if (lead && blockIdx.x == 0) cnt->n_recv = cnt->n_defer = 0;
		d_slope<M, V>(g, P, C, a.B, list, n, a.limiter, epoch0 + 2, cnt);
		if constexpr (M::MULTI) {
			// the sweeps read and write the volume fractions only, which neither slopes nor indicator touch
			d_smooth_alpha<M>(r, P, C, a.B, list, n, nullptr, P.tmp, L, epoch0 + 3, e_upd, cnt);
			if (!run_barrier(a, arrivals, &s_ok)) return;
			d_smooth_alpha<M>(r, P, C, a.B, list, n, P.tmp, P.tmp2, L, epoch0 + 4, e_upd, cnt);
		} else {
			if (!run_barrier(a, arrivals, &s_ok)) return;
		}
		d_estimate<M>(g, P, C, list, n, L, counter_L, epoch0 + EX, s_ls.split, cnt);
		if constexpr (M::MULTI) {
			if (!run_barrier(a, arrivals, &s_ok)) return;
			d_smooth_alpha<M>(g, P, C, a.B, list, n, P.tmp2, P.k + (size_t) M::ALPHAS * P.cap, L, epoch0 + 5, e_upd, cnt);
			if (!run_barrier(a, arrivals, &s_ok)) return;
			d_normal<M>(g, P, C, a.B, list, n, epoch0 + 6, e_upd, cnt);
			if (a.sigma) {
				if (!run_barrier(a, arrivals, &s_ok)) return;
				d_curvature<M>(g, P, C, a.B, list, n, cnt);
				if (!run_barrier(a, arrivals, &s_ok)) return;
				d_smooth_kappa<M>(g, P, C, a.B, list, n, cnt);
				if (!run_barrier(a, arrivals, &s_ok)) return;
				d_store_tmp(g, P, list, n, M::KAPPA, P.tmp);
				// each cell's record takes its own curvature, written by the same thread just above
				d_rec_k<M>(g, P, list, n);
			}
		}
		if (!run_barrier(a, arrivals, &s_ok)) return;
		const int n_split = __ldcg(&cnt->n_split);
		if ((long long) s_top + (long long) NC * n_split + 16 > P.cap) {
			if (lead) s_stop = RUN_CAPACITY;
			__syncthreads();
			break;
		}
		const bool cand = counter_L == 1 && C.coarsen;  // when d_estimate may make candidates
		if (n_split > 0 || cand) {
			// a split cell and the family of a coarsened one have no cell in common
			d_split<M>(g, P, C, &cnt->n_split, s_ls.split, L, s_ls.fresh, epoch0 + EX + 1, cnt);
			if (cand) d_coarsen<M>(r, P, C, list, n, L, s_ls.fresh, epoch0 + EX + 2, cnt);
			if (!run_barrier(a, arrivals, &s_ok)) return;
		}
		// the neighbour repair reads no time level and the reassignment no neighbour
		const int n_new = __ldcg(&cnt->n_new);
		if (n_new > 0) d_nbr_fresh<M>(r, P, C, &cnt->n_new, s_ls.fresh, cnt);
		run_reassign<M>(g, P, C, list, n, L, dtL, counter_L, s_ls, cnt, s_warp);
		d_reassign<M>(g, P, C, s_ls.fresh, &cnt->n_new, 0, L, dtL, counter_L, s_ls, cnt);
		d_flush(r, P, s_ls.buf[L], &cnt->buf[L], s_ls.tmp, &cnt->n_tmp, L, cnt);
		if (!run_barrier(a, arrivals, &s_ok)) return;
		// the substep's end (impl/integrate.hpp:56-67)
		if (lead) {
			int v[MAX_ACTI];
#pragma unroll
			for (int l = 0; l < MAX_ACTI; ++l) v[l] = __ldcg(cnt->clu + l);
			const int n_tmp = __ldcg(&cnt->n_tmp), n_unsplit = __ldcg(&cnt->n_unsplit);
			const uint32_t status = __ldcg(&cnt->status);
			s_top = __ldcg(&cnt->top);
#pragma unroll
			for (int l = 0; l < MAX_ACTI; ++l) s_clu[l] = l == L ? n_tmp : v[l];
			if (blockIdx.x == 0) {
				// the other blocks have the new length in hand and read neither before the next barrier
				cnt->clu[L] = n_tmp;
				cnt->buf[L] = 0;
			}
			int32_t *x     = s_ls.clu[L];
			s_ls.clu[L]    = s_ls.tmp;
			s_ls.tmp       = x;
			s.counter[L]   = (s.counter[L] + 1) % 2;
			s.time[L] += dtL;
			s.epoch += SUBSTEP_EPOCHS<M>;
			s_tot[0] += n_split;
			s_tot[1] += n_unsplit;
			s_tot[2] += n_tmp;
			s_tot[3] += 1;
			if (status) s_stop = RUN_STATUS;
		}
		__syncthreads();
	}
	// the host reads both once the launch is over: no copies to queue behind it
	if (blockIdx.x == 0 && threadIdx.x < 32) {
		const int *src = reinterpret_cast<const int *>(cnt);
		int *dst       = reinterpret_cast<int *>(a.out_cnt);
		for (int w = threadIdx.x; w < (int) (sizeof(Counters) / 4); w += 32) dst[w] = __ldcg(src + w);
		__syncwarp();
		if (lead) {
			RunState &o = *a.out;
			o.sch       = s;
			o.seq       = s_seq;
			o.l         = s_l;
			o.L         = s_L;
			o.splits    = s_tot[0];
			o.unsplits  = s_tot[1];
			o.updates   = s_tot[2];
			o.substeps  = s_tot[3];
			for (int l = 0; l < MAX_ACTI; ++l) o.clu[l] = s_ls.clu[l];
			o.tmp  = s_ls.tmp;
			o.stop = s_stop;
		}
	}
}

}  // namespace dg
