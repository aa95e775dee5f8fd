// Host side of the solver: node-pool management, the Integrator constructor sequence and the ACTI
// level scheduler of Integrator::integrate, issuing the stage kernels of stages.cuh.
#pragma once

#include "mem.cuh"
#include "run.cuh"
#include "solver_base.h"

#include <cub/cub.cuh>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

namespace dg {

inline int grid_for(long long n, int max_blocks = 148 * 16) {
	long long b = (n + BLOCK - 1) / BLOCK;
	if (b < 1) b = 1;
	if (b > max_blocks) b = max_blocks;
	return (int) b;
}
// The same number of threads in blocks of `threads`.
inline int grid_threads(long long n, int threads) { return grid_for(n) * (BLOCK / threads); }

template<class M>
class Batch;

template<class M>
class Solver : public SolverBase {
	static constexpr int D = M::D, E = M::E, NC = 1 << D, NF = 2 * D;
	friend class Batch<M>;

	MemoryUser memory_;
	cudaStream_t st_ = 0;
	Consts C_{};
	BcTable B_{};
	Pool P_{};
	Lists Ls_{};
	Counters *d_cnt_ = nullptr;
	Counters *h_cnt_ = nullptr;  // pinned, behind h_run_ unless a batch holds the counters
	unsigned *d_bar_ = nullptr;  // the grid barrier of device-resident runs
	RunState *h_run_ = nullptr;  // pinned: where a run leaves its schedule state
	int run_cluster_ = 0;        // blocks of a clustered run on this device (0: not asked yet)
	void *pool_mem_  = nullptr;
	void *spare_mem_  = nullptr;  // one field's worth of slots: target of the re-sort and gc permutations
	size_t spare_bytes_ = 0;
	void *sort_mem_  = nullptr;   // keys/values/temp storage of the re-sort
	size_t sort_bytes_ = 0;
	bool resort_     = true;
	void *list_mem_  = nullptr;
	void *bc_mem_    = nullptr;
	double *ff_mem_    = nullptr;  // face fluxes next to receivers (Pool::ff)
	double *du_mem_    = nullptr;  // face-flux sums of the running cluster (Pool::du)
	int32_t *pos_mem_  = nullptr;  // list positions of the running cluster's cells (Pool::pos)
	void *sel_mem_     = nullptr;  // stay marks of the running list and the ordered compaction's temp storage
	size_t sel_tmp_bytes_ = 0;
	int opts_          = DG_OPT_DEFAULT;  // stage implementation choices (DG_OPT_*)
	int32_t *d_leaves_ = nullptr;  // scratch list used at construction
	double *d_read_    = nullptr;
	int32_t *d_readlv_ = nullptr;
	long long read_cap_ = 0;
	int limiter_ = 0;
	int coarsen_every_ = 1;  // global steps between coarsening passes
	bool visc_   = false;  // viscous/heat terms present (multiphase with any non-zero mu or lambda)
	bool mixed_  = false;  // FP32 reconstruction and flux, FP64 update and EOS recovery
	bool sigma_  = false;  // surface tension present

	// scheduler state (integrator/integrator.hpp:46-58)
	int acti_counter_[MAX_ACTI] = {};
	double acti_time_[MAX_ACTI] = {};
	int max_acti_ = 0;
	double global_dt_ = -INFINITY;
	long long n_substeps_ = 0, n_global_ = 0, updates_ = 0, n_gc_ = 0;
	long long n_split_total_ = 0, n_unsplit_total_ = 0;
	int stamp_ = 0;
	int epoch_ = 2;           // kernel epochs of the subtree-mean memo (Pool::mod / Pool::cst)
	int max_tree_level_ = 0;  // deepest tree level any node can reach

	// launch accounting and optional per-kernel event timing
	struct Pending {
		int kind;
		cudaEvent_t a, b;
		long long cells;
	};
	bool prof_ = false;
	std::vector<cudaEvent_t> ev_free_;
	std::vector<Pending> pending_;
	double kms_[DG_NK]          = {};
	long long klaunch_[DG_NK]   = {};
	long long kcells_[DG_NK]    = {};
	long long n_launches_       = 0;

	cudaEvent_t get_event() {
		if (ev_free_.empty()) {
			cudaEvent_t e;
			DG_CUDA(cudaEventCreate(&e));
			return e;
		}
		cudaEvent_t e = ev_free_.back();
		ev_free_.pop_back();
		return e;
	}

	template<class Fn>
	void run_k(int kind, long long cells, Fn &&fn) {
		cudaEvent_t a = nullptr, b = nullptr;
		if (prof_) {
			a = get_event();
			b = get_event();
			DG_CUDA(cudaEventRecord(a, st_));
		}
		fn();
		n_launches_++;
		klaunch_[kind]++;
		kcells_[kind] += cells;
		if (prof_) {
			DG_CUDA(cudaEventRecord(b, st_));
			pending_.push_back({kind, a, b, cells});
		}
	}

	void drain_events() {
		for (auto &p: pending_) {
			float ms = 0.f;
			DG_CUDA(cudaEventElapsedTime(&ms, p.a, p.b));
			kms_[p.kind] += ms;
			ev_free_.push_back(p.a);
			ev_free_.push_back(p.b);
		}
		pending_.clear();
	}

public:
	void set_profiling(bool on) override { prof_ = on; }
	void set_options(int opts) override { opts_ = opts; }
	void set_form(int form) override {
		if (form != DG_FORM_FP64 && form != DG_FORM_MIXED) throw dg_error(DG_ERR_ARG, "unknown form");
		mixed_ = form == DG_FORM_MIXED;
	}

	explicit Solver(const dg_case &c) {
		limiter_ = c.limiter;
		setup_consts(c);
		upload_bcs(c);
		long long cap = (long long) c.n_nodes + c.n_nodes / 2 + 1024;
		if (c.params[DG_P_POOL_CAP] > 0) cap = std::max((long long) c.params[DG_P_POOL_CAP], (long long) c.n_nodes + 1024);
		if (cap > 2000000000LL) throw dg_error(DG_ERR_CAPACITY, "node pool capacity above 2e9 slots");
		alloc_pool((int) cap);
		alloc_lists(cap);
		DG_CUDA(mem_alloc((void **) &d_cnt_, sizeof(Counters), st_));
		static_assert(sizeof(RunState) + 16 + sizeof(Counters) <= PINNED_BYTES, "run state and counters share a pinned block");
		DG_CUDA(pinned_alloc((void **) &h_run_));
		h_cnt_ = (Counters *) (h_run_ + 1);
		DG_CUDA(cudaMemset(d_cnt_, 0, sizeof(Counters)));
		DG_CUDA(mem_alloc((void **) &d_bar_, sizeof(unsigned), st_));
		upload_tree(c);
		construct();
	}

	~Solver() override {
		cudaStreamSynchronize(st_);
		mem_free_idle(pool_mem_);
		mem_free_idle(spare_mem_);
		mem_free_idle(sort_mem_);
		mem_free_idle(list_mem_);
		mem_free_idle(bc_mem_);
		mem_free_idle(ff_mem_);
		mem_free_idle(du_mem_);
		mem_free_idle(sel_mem_);
		mem_free_idle(pos_mem_);
		mem_free_idle(d_cnt_);
		mem_free_idle(d_bar_);
		pinned_release(h_run_);
		mem_free_idle(d_leaves_);
		mem_free_idle(d_read_);
		mem_free_idle(d_readlv_);
		if (owned_stream_) cudaStreamDestroy(owned_stream_);
		for (auto e: ev_free_) cudaEventDestroy(e);
		for (auto &p: pending_) {
			cudaEventDestroy(p.a);
			cudaEventDestroy(p.b);
		}
	}

	void set_stream(cudaStream_t s) override { st_ = s; }

	cudaStream_t owned_stream_ = nullptr;
	void own_stream() override {
		if (st_ != 0) return;
		if (!owned_stream_) DG_CUDA(cudaStreamCreateWithFlags(&owned_stream_, cudaStreamNonBlocking));
		st_ = owned_stream_;
	}

	// ---------------------------------------------------------------------------------------
	void setup_consts(const dg_case &c) {
		const double *pr = c.params;
		C_.side = pr[DG_P_SIDE];
		for (int d = 0; d < 3; ++d) {
			C_.active[d]   = pr[DG_P_ACTIVE0 + d];
			C_.periodic[d] = pr[DG_P_PERIODIC0 + d] != 0.0;
		}
		C_.max_cfl              = pr[DG_P_MAX_CFL];
		C_.min_err              = pr[DG_P_MIN_ERR];
		C_.max_err              = pr[DG_P_MAX_ERR];
		C_.max_refinement_level = (int) pr[DG_P_MAX_LEVEL];
		max_dt_cfg_             = pr[DG_P_MAX_DT];
		pruned_                 = (long long) pr[DG_P_PRUNED];
		for (int q = 0; q < E; ++q) C_.weights[q] = c.weights[q];
		ModelConsts &m = C_.m;
		m.ns_mu = pr[DG_P_NS_MU];
		m.ns_lambda = pr[DG_P_NS_LAMBDA];
		m.gamma1 = pr[DG_P_GAMMA1];
		m.gamma2 = pr[DG_P_GAMMA2];
		m.P1 = pr[DG_P_P1];
		m.P2 = pr[DG_P_P2];
		m.cp1 = pr[DG_P_CP1];
		m.cp2 = pr[DG_P_CP2];
		m.cv1 = pr[DG_P_CV1];
		m.cv2 = pr[DG_P_CV2];
		m.mu1 = pr[DG_P_MU1];
		m.mu2 = pr[DG_P_MU2];
		m.lambda1 = pr[DG_P_LAMBDA1];
		m.lambda2 = pr[DG_P_LAMBDA2];
		m.sigma = pr[DG_P_SIGMA];
		{
			const double g1 = m.gamma1, g2 = m.gamma2;
			m.eos[0] = 1 / (g1 - 1) - 1 / (g2 - 1), m.eos[1] = g1 * m.P1 / (g1 - 1), m.eos[2] = g2 * m.P2 / (g2 - 1);
			const float f1 = (float) g1, f2 = (float) g2;
			m.eos_f[0] = 1 / (f1 - 1) - 1 / (f2 - 1), m.eos_f[1] = f1 * (float) m.P1 / (f1 - 1), m.eos_f[2] = f2 * (float) m.P2 / (f2 - 1);
		}
		if constexpr (M::MULTI) visc_ = m.mu1 != 0.0 || m.mu2 != 0.0 || m.lambda1 != 0.0 || m.lambda2 != 0.0;
		else visc_ = M::VISC;
		sigma_ = m.sigma != 0.0;
		C_.visc = visc_ ? 1 : 0;
		if (c.n_zones > MAX_ZONES) throw dg_error(DG_ERR_ARG, "too many refinement zones");
		C_.n_zones = c.n_zones;
		C_.coarsen = 1;
		for (int z = 0; z < c.n_zones; ++z) {
			for (int d = 0; d < 3; ++d) {
				C_.zx0[z][d] = c.zones[7 * z + d];
				C_.zx1[z][d] = c.zones[7 * z + 3 + d];
			}
			C_.zlevel[z] = (int) c.zones[7 * z + 6];
		}
		// Per-level size (exact halving from the root, integrator/domain.hpp:207), and volume/area
		// evaluated with the same std::pow calls as Cell::volume / CellFace::area
		// (integrator/cell.hpp:575-577, 622-624).
		double s = C_.side;
		for (int l = 0; l < MAX_TREE; ++l) {
			C_.size[l] = s;
			C_.vol[l]  = std::pow(s, D);
			C_.area[l] = std::pow(s, D - 1);
			for (int d = 0; d < 3; ++d) {
				if (d >= D) {
					C_.a0[l][d] = 0;
					C_.na[l][d] = 1;
					continue;
				}
				// active box [-A/2, A/2] in cells of level l of the root box [-S/2, S/2]
				double cells = C_.active[d] / s;
				double off   = 0.5 * (C_.side - C_.active[d]) / s;
				long long nc = std::llround(cells), oc = std::llround(off);
				C_.na[l][d]  = (int) nc;
				C_.a0[l][d]  = (int) oc;
				if (l >= (int) pr[DG_P_MIN_LEVEL] && (std::fabs(cells - nc) > 1e-9 || std::fabs(off - oc) > 1e-9))
					throw dg_error(DG_ERR_UNSUPPORTED, "active box not aligned with the cell grid at the base level");
			}
			s = 0.5 * s;
		}
	}

	void upload_bcs(const dg_case &c) {
		int n        = c.n_bc > 0 ? c.n_bc : 1;
		size_t bytes = sizeof(int) * n + sizeof(double) * n * (E + D + 1) + 1024;
		DG_CUDA(mem_alloc((void **) &bc_mem_, bytes, st_));
		char *b   = (char *) bc_mem_;
		int *type = (int *) b;
		b += ((sizeof(int) * n + 255) / 256) * 256;
		double *pin = (double *) b;
		double *nrm = pin + (size_t) n * E;
		double *fad = nrm + (size_t) n * D;
		if (c.n_bc > 0) {
			DG_CUDA(cudaMemcpy(type, c.bc_type, sizeof(int) * c.n_bc, cudaMemcpyHostToDevice));
			DG_CUDA(cudaMemcpy(pin, c.bc_p_in, sizeof(double) * c.n_bc * E, cudaMemcpyHostToDevice));
			DG_CUDA(cudaMemcpy(nrm, c.bc_normal, sizeof(double) * c.n_bc * D, cudaMemcpyHostToDevice));
			DG_CUDA(cudaMemcpy(fad, c.bc_fade_in, sizeof(double) * c.n_bc, cudaMemcpyHostToDevice));
		}
		B_ = BcTable{c.n_bc, type, pin, nrm, fad};
	}

	// ---------------------------------------------------------------------------------------
	// Node pool: every field is an array of `cap` entries per component.
	struct Field {
		void **ptr;
		size_t elem;
		int comps;
		int link = 0;  // holds slot numbers
		int stay = 0;  // scratch of one substep, or marks that no later value equals: need not follow their slots
	};

	std::vector<Field> fields(Pool &P) {
		return {
		    {(void **) &P.parent, 4, 1, 1}, {(void **) &P.child, 4, NC, 1}, {(void **) &P.level, 1, 1},
		    {(void **) &P.acti, 1, 1}, {(void **) &P.clu, 1, 1}, {(void **) &P.flags, 4, 1},
		    {(void **) &P.coord, 4, D}, {(void **) &P.nbr, 4, NF, 1}, {(void **) &P.bc, 2, NF},
		    {(void **) &P.center, 8, D}, {(void **) &P.t, 8, 1}, {(void **) &P.u, 8, E},
		    {(void **) &P.p, 8, E}, {(void **) &P.rec, 8 * Rec<M>::W, 1}, {(void **) &P.avg, 8 * Avg<M>::W, 1},
		    {(void **) &P.mod, 4, 1}, {(void **) &P.cst, 4, 1}, {(void **) &P.avga, 8, 1}, {(void **) &P.csta, 4, 1},
		    {(void **) &P.k, 8, M::P}, {(void **) &P.tslope, 8, visc_ ? M::G : -1},
		    {(void **) &P.grad, 8, visc_ ? D * M::G : -1},
		    {(void **) &P.flux, 8, M::F}, {(void **) &P.err, 8, 1}, {(void **) &P.maxdt, 8, 1},
		    {(void **) &P.cfl, 8, 1}, {(void **) &P.stamp, 4, 1, 0, 1}, {(void **) &P.op, 1, 1},
		    {(void **) &P.tmp, 8, 1, 0, 1}, {(void **) &P.tmp2, 8, 1, 0, 1},
		};
	}

	static size_t align_up(size_t x) { return (x + 255) & ~size_t(255); }

	// The spare buffer of the re-sort and gc holds the largest field of the pool (the reconstruction records,
	// in practice), or a second pool where that is small and fits: a re-sort then writes every field once, in
	// three launches, and the two change places. Field by field it is some seventy launches (0.2 ms, which small trees
	// notice) and every field is written twice (nine trees of a million cells on one level, 0.9 GB of pool each, 35 ms a
	// step against 32). A larger pool's memory is worth more. A solver gives the second pool up again once more than half
	// of the device's memory is in use.
	static constexpr size_t SECOND_POOL_MAX = size_t(1) << 30;
	bool spare_dirty_ = true;   // the spare buffer holds something else than an earlier state of the pool
	bool spare_small_ = false;  // a second pool of this size did not fit
	size_t pool_bytes(Pool &P) {
		size_t total = 0;
		for (auto &f: fields(P)) total += field_bytes(f, P.cap);
		return total;
	}
	bool second_pool() { return spare_bytes_ >= pool_bytes(P_); }
	void ensure_spare() {
		size_t field = 0;
		for (auto &f: fields(P_)) field = std::max(field, field_bytes(f, P_.cap));
		const size_t whole = pool_bytes(P_);
		const bool two     = whole <= SECOND_POOL_MAX && !spare_small_ && !mem_tight(spare_bytes_ >= whole ? 0 : whole);
		if (spare_mem_ && spare_bytes_ >= (two ? whole : field) && (two || spare_bytes_ < whole)) return;
		mem_free(spare_mem_, st_);
		spare_mem_    = nullptr;
		spare_bytes_  = 0;
		spare_dirty_  = true;
		cudaError_t e = mem_alloc((void **) &spare_mem_, two ? whole : field, st_);
		spare_bytes_  = two ? whole : field;
		if (two && e == cudaErrorMemoryAllocation) {
			cudaGetLastError();
			spare_small_ = true;
			e            = mem_alloc((void **) &spare_mem_, field, st_);
			spare_bytes_ = field;
		}
		if (e != cudaSuccess) spare_mem_ = nullptr, spare_bytes_ = 0;
		DG_CUDA(e);
	}

	// Bytes of one field: comps < 0 marks a field this case does not store (no storage, null pointer);
	// a model without components of a field (comps 0) still gets one.
	static size_t field_bytes(const Field &f, int cap) {
		return f.comps < 0 ? 0 : align_up(f.elem * (size_t) cap * (f.comps > 0 ? f.comps : 1));
	}

	void place_fields(Pool &P, void *mem) {
		char *b = (char *) mem;
		for (auto &f: fields(P)) {
			*f.ptr = f.comps < 0 ? nullptr : b;
			b += field_bytes(f, P.cap);
		}
	}

	void *carve_pool(Pool &P, int cap) {
		P.cap              = cap;
		const size_t total = pool_bytes(P);
		void *mem          = nullptr;
		DG_CUDA(mem_alloc((void **) &mem, total, st_));
		DG_CUDA(cudaMemsetAsync(mem, 0, total, st_));
		place_fields(P, mem);
		return mem;
	}

	void alloc_pool(int cap) {
		pool_mem_ = carve_pool(P_, cap);
		alloc_derived(cap);
	}

	// Per-substep scratch. By pool slot: pos (a running-cluster cell's list position). By list position,
	// sized to the largest list a substep has run so far (grown by a quarter when a larger one comes):
	// receiver face fluxes and face-flux sums.
	void alloc_derived(int cap) {
		mem_free(pos_mem_, st_);
		pos_mem_ = nullptr;
		DG_CUDA(mem_alloc((void **) &pos_mem_, sizeof(int32_t) * (size_t) cap, st_));
		attach_derived();
	}

	long long scratch_cap_ = 0;
	void ensure_scratch(long long n) {
		if (n <= scratch_cap_) return;
		const long long want = std::max(std::max(n, scratch_cap_ + scratch_cap_ / 4), 1024LL);
		mem_free(ff_mem_, st_);
		mem_free(du_mem_, st_);
		mem_free(sel_mem_, st_);
		ff_mem_      = nullptr;
		du_mem_      = nullptr;
		sel_mem_     = nullptr;
		scratch_cap_ = 0;
		DG_CUDA(mem_alloc((void **) &ff_mem_, sizeof(double) * M::F * NF * (size_t) want, st_));
		DG_CUDA(mem_alloc((void **) &du_mem_, (sizeof(double) * M::F + sizeof(int32_t)) * (size_t) want, st_));
		// stay marks (one byte per list position, rounded to 256) followed by the temp storage of the
		// order-keeping compaction of `want` items
		sel_tmp_bytes_ = 0;
		DG_CUDA(cub::DeviceSelect::Flagged(nullptr, sel_tmp_bytes_, (const int32_t *) nullptr, (const uint8_t *) nullptr,
		                                   (int32_t *) nullptr, (int *) nullptr, (int) want, st_));
		DG_CUDA(mem_alloc((void **) &sel_mem_, stay_bytes(want) + sel_tmp_bytes_, st_));
		scratch_cap_ = want;
		attach_derived();
	}

	static size_t stay_bytes(long long want) { return ((size_t) want + 255) / 256 * 256; }
	uint8_t *stay_marks() const { return static_cast<uint8_t *>(sel_mem_); }

	void attach_derived() {
		P_.ff   = ff_mem_;
		P_.du    = du_mem_;
		P_.dmask = (int32_t *) (du_mem_ + (size_t) M::F * (size_t) scratch_cap_);
		P_.pos  = pos_mem_;
	}

	// The capacity a pool grows to when `need` slots must fit and `want` would be chosen: `want` when the
	// new pool and lists fit in the free device memory (counting the scratch, spare buffer and sort keys
	// that grow_pool releases first, less 1 GiB), else as many slots as fit, and never fewer than `need`.
	long long growth_target(long long need, long long want) {
		size_t free_b = 0, total_b = 0;
		DG_CUDA(cudaMemGetInfo(&free_b, &total_b));
		const size_t released = sizeof(double) * M::F * (NF + 1) * (size_t) scratch_cap_ + spare_bytes_ + sort_bytes_;
		size_t per_slot = sizeof(int32_t) * (2 * MAX_ACTI + 5);
		for (auto &f: fields(P_))
			if (f.comps >= 0) per_slot += f.elem * (size_t) (f.comps > 0 ? f.comps : 1);
		const long long avail = (long long) (free_b + mem_unused() + released) - (1LL << 30);
		const long long fit   = avail > 0 ? avail / (long long) per_slot : 0;
		return std::max(need, std::min(want, fit));
	}

	// The rows of field f from `src` (component stride src_cap) to `dst`.
	static void add_rows(RowTable &t, const Field &f, const void *src, int src_cap, void *dst, int dst_cap, bool relink) {
		for (int c = 0; c < f.comps; ++c)
			t.r[t.n++] = {(const char *) src + f.elem * (size_t) src_cap * c, (char *) dst + f.elem * (size_t) dst_cap * c,
			              (int) f.elem, relink && f.link};
	}

	// Grows the node pool: a new pool of new_cap slots takes every field, then the old one goes. Grows
	// between the indicator and the split of a substep, when the stages that use the list scratch are
	// done, so the scratch, the spare buffer and the re-sort keys are released first (they come back at
	// their next use) and the peak holds the two pools and the lists only.
	void grow_pool(int new_cap) {
		DG_CUDA(cudaStreamSynchronize(st_));
		mem_free(spare_mem_, st_);
		spare_mem_   = nullptr;
		spare_bytes_ = 0;
		spare_dirty_ = true;
		spare_small_ = false;
		mem_free(sort_mem_, st_);
		sort_mem_   = nullptr;
		sort_bytes_ = 0;
		mem_free(ff_mem_, st_);
		mem_free(du_mem_, st_);
		mem_free(sel_mem_, st_);
		ff_mem_      = nullptr;
		du_mem_      = nullptr;
		sel_mem_     = nullptr;
		scratch_cap_ = 0;
		attach_derived();
		Pool NP{};
		void *mem = carve_pool(NP, new_cap);
		// the slots in use; the rest of the new pool is zero, as it was in the old one
		auto fo = fields(P_), fn = fields(NP);
		const int used = std::min(h_cnt_->top, P_.cap);
		RowTable t{};
		for (size_t k = 0; k < fo.size(); ++k) {
			if (fo[k].comps <= 0) continue;
			if (fo[k].elem > 8)
				DG_CUDA(cudaMemcpyAsync(*fn[k].ptr, *fo[k].ptr, fo[k].elem * (size_t) used, cudaMemcpyDeviceToDevice, st_));
			else
				add_rows(t, fo[k], *fo[k].ptr, P_.cap, *fn[k].ptr, new_cap, false);
		}
		k_rows<<<dim3(grid_for(used, 148 * 4), t.n), BLOCK, 0, st_>>>(t, used, nullptr, nullptr);
		DG_CUDA(cudaGetLastError());
		mem_free(pool_mem_, st_);
		pool_mem_ = mem;
		P_        = NP;
		alloc_derived(new_cap);
		// lists grow with the pool
		Lists old = Ls_;
		void *old_mem = list_mem_;
		int old_cap   = list_cap_;
		alloc_lists(new_cap);
		auto keep = [&](int32_t *dst, const int32_t *src, int n) {
			if (n > 0) DG_CUDA(cudaMemcpyAsync(dst, src, sizeof(int32_t) * std::min(n, old_cap), cudaMemcpyDeviceToDevice, st_));
		};
		for (int l = 0; l < MAX_ACTI; ++l) {
			keep(Ls_.clu[l], old.clu[l], h_cnt_->clu[l]);
			keep(Ls_.buf[l], old.buf[l], h_cnt_->buf[l]);
		}
		// the pool can grow between the indicator and the split, whose requests are the only list of a
		// substep in use there
		keep(Ls_.split, old.split, h_cnt_->n_split);
		mem_free(old_mem, st_);
	}

	int list_cap_ = 0;
	void alloc_lists(int cap) {
		const int nlists = 2 * MAX_ACTI + 5;
		size_t one       = align_up(sizeof(int32_t) * (size_t) cap);
		DG_CUDA(mem_alloc((void **) &list_mem_, one * nlists, st_));
		char *b = (char *) list_mem_;
		for (int l = 0; l < MAX_ACTI; ++l) {
			Ls_.clu[l] = (int32_t *) b;
			b += one;
			Ls_.buf[l] = (int32_t *) b;
			b += one;
		}
		Ls_.tmp     = (int32_t *) b;
		b += one;
		Ls_.recv    = (int32_t *) b;
		b += one;
		Ls_.split   = (int32_t *) b;
		b += one;
		Ls_.unsplit = (int32_t *) b;
		b += one;
		Ls_.fresh   = (int32_t *) b;
		list_cap_   = cap;
	}

	// ---------------------------------------------------------------------------------------
	// Rows of `comps` values per node into the pool, through a device buffer that holds the largest field.
	template<class To, class From>
	void upload_rows(To *dst, const From *src, int n, int comps, void *buf) {
		if (n <= 0 || comps <= 0) return;
		DG_CUDA(cudaMemcpyAsync(buf, src, sizeof(From) * (size_t) n * comps, cudaMemcpyHostToDevice, st_));
		k_take_rows<From, To><<<grid_for((long long) n * comps), BLOCK, 0, st_>>>((const From *) buf, dst, n, comps, P_.cap);
		DG_CUDA(cudaGetLastError());
	}

	std::vector<int32_t> active_leaves_;

	void upload_tree(const dg_case &c) {
		const int n = c.n_nodes;
		DG_CUDA(cudaStreamSynchronize(st_));
		max_tree_level_ = C_.max_refinement_level;
		for (int z = 0; z < C_.n_zones; ++z) max_tree_level_ = std::max(max_tree_level_, C_.zlevel[z]);
		int deepest = 0;
		for (int i = 0; i < n; ++i) deepest = std::max(deepest, (int) c.level[i]);
		max_tree_level_ = std::max(max_tree_level_, deepest);
		void *buf = nullptr;
		DG_CUDA(mem_alloc(&buf, 8 * (size_t) std::max({NC, NF, D, E}) * (size_t) std::max(n, 1), st_));
		upload_rows(P_.parent, c.parent, n, 1, buf);
		upload_rows(P_.child, c.children, n, NC, buf);
		upload_rows(P_.level, c.level, n, 1, buf);
		upload_rows(P_.flags, (const uint32_t *) c.flags, n, 1, buf);
		upload_rows(P_.bc, c.bc, n, NF, buf);
		upload_rows(P_.center, c.center, n, D, buf);
		upload_rows(P_.p, c.p, n, E, buf);
		mem_free(buf, st_);
		DG_CUDA(cudaMemsetAsync(P_.acti, 0xff, n, st_));  // -1
		DG_CUDA(cudaMemsetAsync(P_.clu, 0xff, n, st_));   // CLU_NONE
		// integer coordinates, parents before children
		for (int l = 1; l <= deepest; ++l) k_coords<D><<<grid_for(n), BLOCK, 0, st_>>>(P_, n, l);
		// Node::error as the scene leaves it: -1 on every split child (integrator/domain.hpp:215), kept by
		// leaves that never get an estimate (inactive ones) and summed by unsplit (domain.hpp:306-309)
		k_fill_f64<<<grid_for(n), BLOCK, 0, st_>>>(P_.err, -1.0, n);
		DG_CUDA(cudaGetLastError());
		active_leaves_.clear();
		for (int i = 1; i < n; ++i)
			if ((c.flags[i] & DG_F_LEAF) && (c.flags[i] & DG_F_ACTIVE)) active_leaves_.push_back(i);
		int coarsest = MAX_TREE;
		for (int i: active_leaves_) coarsest = std::min(coarsest, (int) c.level[i]);
		h_cnt_->top      = n;
		h_cnt_->coarsest = coarsest;
		DG_CUDA(cudaMemcpy(&d_cnt_->top, &n, sizeof(int), cudaMemcpyHostToDevice));
		DG_CUDA(cudaMemcpy(&d_cnt_->coarsest, &coarsest, sizeof(int), cudaMemcpyHostToDevice));
	}

	// Integrator constructor body (integrator/integrator.hpp:100-160).
	void construct() {
		const int n = (int) active_leaves_.size();
		DG_CUDA(mem_alloc((void **) &d_leaves_, sizeof(int32_t) * (n > 0 ? n : 1), st_));
		DG_CUDA(cudaMemcpy(d_leaves_, active_leaves_.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice));
		const int g = grid_for(n);
		k_init_cells<M><<<g, BLOCK, 0, st_>>>(P_, C_, d_leaves_, n, d_cnt_);
		k_nbr_init<M><<<g, BLOCK, 0, st_>>>(P_, C_, d_leaves_, n);
		// every memo starts stale: mod = 1 > cst = 0
		k_fill_i32<<<grid_for(P_.cap), BLOCK, 0, st_>>>(P_.mod, 1, P_.cap);
		// neighbour values and slopes of every leaf, in pieces of the scratch's size
		ensure_scratch(std::max(n / 2, 1));
		for (int off = 0; off < n; off += (int) scratch_cap_) launch_slope(d_leaves_ + off, std::min<int>(n - off, (int) scratch_cap_));
		if constexpr (M::MULTI) multiphase_aux(d_leaves_, n, -1, 0);
		DG_CUDA(cudaGetLastError());
		sync_counters();
		global_dt_ = std::fmax(-INFINITY, h_cnt_->dmax);
		global_dt_ = std::min(0.9 * global_dt_, max_dt_cfg());
		k_assign<M><<<g, BLOCK, 0, st_>>>(P_, C_, d_leaves_, n, global_dt_, Ls_, d_cnt_);
		DG_CUDA(cudaGetLastError());
		sync_counters();
		check_status();
		mem_free(d_leaves_, st_);  // the constructor's list of every leaf is not used again
		d_leaves_ = nullptr;
		max_acti_ = 0;
		for (int l = 0; l < MAX_ACTI; ++l)
			if (h_cnt_->clu[l] > 0) max_acti_ = std::max(max_acti_, l);
	}

	double max_dt_cfg_ = 1.0;
	double max_dt_cfg() const { return max_dt_cfg_; }
	long long pruned_ = 0;  // node slots the host left out of the upload; part of the reference's tree size

	// The garbage-collection trigger of impl/integrate.hpp:78-84: active leaves in clusters below a fifth
	// of tree.size() - 1, the tree size counting the slots left out of the upload.
	bool gc_due() const {
		long long n_in = 0;
		for (int l = 0; l < MAX_ACTI; ++l) n_in += h_cnt_->clu[l];
		return (double) n_in / (double) (h_cnt_->top - 1 + pruned_) < 0.2;
	}

public:
	void set_max_dt(double v) { max_dt_cfg_ = v; }

private:
	// smooth_alpha x3, normal_update, curvature_update, smooth_curvature over one cell list
	// (impl/integrate.hpp:284-289, integrator/integrator.hpp:134-143).
	// Lm: the ACTI level whose cluster `list` is, or -1 when the list holds every leaf (constructor).
	// e_upd: epoch of the substep's cell update (0: no memoised volume-fraction means).
	void multiphase_aux(const int32_t *list, int n, int Lm, int e_upd) {
		if constexpr (M::MULTI) {
			constexpr int G = NF <= 4 ? 4 : 8;
			const int g  = grid_for(n);
			const int gl = grid_for((long long) n * G);
			double *alphas = P_.k + (size_t) M::ALPHAS * P_.cap;
			run_k(DG_K_AUX, n, [&] {
				k_smooth_alpha<M><<<gl, BLOCK, 0, st_>>>(P_, C_, B_, list, n, nullptr, P_.tmp, Lm, ++epoch_, e_upd, d_cnt_);
			});
			run_k(DG_K_AUX, n, [&] {
				k_smooth_alpha<M><<<gl, BLOCK, 0, st_>>>(P_, C_, B_, list, n, P_.tmp, P_.tmp2, Lm, ++epoch_, e_upd, d_cnt_);
			});
			run_k(DG_K_AUX, n, [&] {
				k_smooth_alpha<M><<<gl, BLOCK, 0, st_>>>(P_, C_, B_, list, n, P_.tmp2, alphas, Lm, ++epoch_, e_upd, d_cnt_);
			});
			run_k(DG_K_AUX, n, [&] { k_normal<M><<<gl, BLOCK, 0, st_>>>(P_, C_, B_, list, n, ++epoch_, e_upd, d_cnt_); });
			// The curvature only enters through sigma * kappa (model/multi.hpp:142, 216, 190-193); without
			// surface tension those products are zeros and the curvature stages are skipped.
			if (sigma_) {
				run_k(DG_K_AUX, n, [&] { k_curvature<M><<<g, BLOCK, 0, st_>>>(P_, C_, B_, list, n, d_cnt_); });
				run_k(DG_K_AUX, n, [&] { k_smooth_kappa<M><<<g, BLOCK, 0, st_>>>(P_, C_, B_, list, n, d_cnt_); });
				run_k(DG_K_AUX, n, [&] { k_store_tmp<<<g, BLOCK, 0, st_>>>(P_, list, n, M::KAPPA, P_.tmp); });
				run_k(DG_K_AUX, n, [&] { k_rec_k<M><<<g, BLOCK, 0, st_>>>(P_, list, n); });
			}
		}
	}

	// Face-flux sums of the running cluster into du, receivers of slower clusters into Ls_.recv.
	void launch_face_sum(const int32_t *list, int n, int L, double dtL, int stamp) {
		constexpr int G = NF <= 4 ? 4 : 8, T = FACE_THREADS;
		if (opts_ & DG_OPT_FACE_TILES) {
			constexpr int TC = FaceTile<M>::TC;
			const int gt = (int) std::max<long long>(1, ((long long) n + TC - 1) / TC);
			if (mixed_) {
				if (visc_) k_face_tile<M, true, float><<<gt, T, 0, st_>>>(P_, C_, B_, list, n, L, dtL, stamp, Ls_.recv, Ls_.fresh, d_cnt_);
				else k_face_tile<M, false, float><<<gt, T, 0, st_>>>(P_, C_, B_, list, n, L, dtL, stamp, Ls_.recv, Ls_.fresh, d_cnt_);
			} else {
				if (visc_) k_face_tile<M, true, double><<<gt, T, 0, st_>>>(P_, C_, B_, list, n, L, dtL, stamp, Ls_.recv, Ls_.fresh, d_cnt_);
				else k_face_tile<M, false, double><<<gt, T, 0, st_>>>(P_, C_, B_, list, n, L, dtL, stamp, Ls_.recv, Ls_.fresh, d_cnt_);
			}
			return;
		}
		const int g = grid_threads((long long) n * G, T);
		if (mixed_) {
			if (visc_) k_face_sum<M, true, float><<<g, T, 0, st_>>>(P_, C_, B_, list, n, L, dtL, stamp, Ls_.recv, Ls_.fresh, d_cnt_);
			else k_face_sum<M, false, float><<<g, T, 0, st_>>>(P_, C_, B_, list, n, L, dtL, stamp, Ls_.recv, Ls_.fresh, d_cnt_);
		} else {
			if (visc_) k_face_sum<M, true, double><<<g, T, 0, st_>>>(P_, C_, B_, list, n, L, dtL, stamp, Ls_.recv, Ls_.fresh, d_cnt_);
			else k_face_sum<M, false, double><<<g, T, 0, st_>>>(P_, C_, B_, list, n, L, dtL, stamp, Ls_.recv, Ls_.fresh, d_cnt_);
		}
	}

	// Slopes, Hancock rhs and (viscous) gradients of a cell list.
	void launch_slope(const int32_t *list, int n) {
		constexpr int G = NF <= 4 ? 4 : 8, T = SLOPE_THREADS;
		const int g = grid_threads((long long) n * G, T);
		if (visc_) k_slope<M, true><<<g, T, 0, st_>>>(P_, C_, B_, list, n, limiter_, ++epoch_, d_cnt_);
		else k_slope<M, false><<<g, T, 0, st_>>>(P_, C_, B_, list, n, limiter_, ++epoch_, d_cnt_);
	}

	void sync_counters() {
		DG_CUDA(cudaMemcpyAsync(h_cnt_, d_cnt_, sizeof(Counters), cudaMemcpyDeviceToHost, st_));
		DG_CUDA(cudaStreamSynchronize(st_));
		drain_events();
	}

	void check_status() {
		uint32_t s = h_cnt_->status & ~ST_NAN;
		if (s & ST_CAPACITY) throw dg_error(DG_ERR_CAPACITY, "device list or pool capacity exceeded");
		if (s & ST_DEPTH) throw dg_error(DG_ERR_DEPTH, "tree level jump deeper than supported");
		if (s & ST_MISSING_BC) throw dg_error(DG_ERR_MISSING_BC, "face without neighbour or boundary condition");
		if (s & ST_SPLIT_UNSPLIT) throw dg_error(DG_ERR_UNSUPPORTED, "cell both split and coarsened in one substep");
	}

	// One ACTI-level substep: impl/integrate.hpp:277-299 minus the host bookkeeping. The head runs up to
	// the indicator, the tail regrids and rebuilds the cluster's list.
	void substep_head(int L) {
		const int n      = h_cnt_->clu[L];
		const double dtL = global_dt_ / (double) (1 << L);
		ensure_scratch(n);
		// A split takes 2^D new slots. When the pool cannot take a split of every cluster cell, the
		// split requests are read back after the indicator and the pool grown to fit them.
		const bool tight = (long long) h_cnt_->top + (long long) NC * n + 16 > P_.cap;
		const int stamp_recv = ++stamp_;
		// n_recv .. status
		DG_CUDA(cudaMemsetAsync(&d_cnt_->n_recv, 0, (char *) (&d_cnt_->status + 1) - (char *) &d_cnt_->n_recv, st_));
		const int g        = grid_for(n);
		int32_t *list      = Ls_.clu[L];
		const int counterL = acti_counter_[L];

		constexpr int LPC = NF <= 4 ? 4 : 8;  // receive lanes per cell
		int e_upd = 0;                       // epoch of this substep's cell update
		run_k(DG_K_FLUX, n, [&] { launch_face_sum(list, n, L, dtL, stamp_recv); });
		run_k(DG_K_RECV, 0, [&] {
			e_upd       = ++epoch_;
			const int gr = grid_for((long long) n * LPC);
			if (mixed_) k_flux_receive<M, float><<<gr, BLOCK, 0, st_>>>(P_, Ls_.recv, list, Ls_.fresh, n, L, e_upd, d_cnt_);
			else k_flux_receive<M, double><<<gr, BLOCK, 0, st_>>>(P_, Ls_.recv, list, Ls_.fresh, n, L, e_upd, d_cnt_);
		});
		run_k(DG_K_UPDATE, n, [&] {
			if (visc_) k_update<M, true><<<g, BLOCK, 0, st_>>>(P_, C_, list, n, dtL, d_cnt_);
			else k_update<M, false><<<g, BLOCK, 0, st_>>>(P_, C_, list, n, dtL, d_cnt_);
		});
		run_k(DG_K_SLOPE, n, [&] { launch_slope(list, n); });
		if constexpr (M::MULTI) multiphase_aux(list, n, L, e_upd);
		run_k(DG_K_ESTIMATE, n, [&] {
			constexpr int GE = NF <= 4 ? 4 : 8;
			k_estimate<M><<<grid_for((long long) n * GE), BLOCK, 0, st_>>>(P_, C_, list, n, L, counterL, ++epoch_, Ls_.split,
			                                                                 d_cnt_);
		});
		if (tight) {
			sync_counters();
			check_status();
			grow_for_splits();
		}
	}

	// A pool with room for the split requests that the host's counters hold.
	void grow_for_splits() {
		const long long need = (long long) h_cnt_->top + (long long) NC * h_cnt_->n_split + 16;
		if (need <= P_.cap) return;
		const long long want = growth_target(need, grown(need));
		grow_pool((int) std::min<long long>(want, 2000000000LL));
	}

	// The capacity wanted when `need` slots must fit: a quarter more, and twice the old one while that is small
	// (a growth costs about 0.3 ms whatever the size, and a tree that refines from a coarse grid grows ten times
	// its size within a few steps).
	static constexpr size_t DOUBLING_MAX = size_t(512) << 20;
	long long grown(long long need) {
		const long long cap = P_.cap;
		return std::max(need + need / 4, pool_bytes(P_) < DOUBLING_MAX ? cap * 2 : cap * 5 / 4);
	}

	void substep_tail(int L, int n) {
		const double dtL   = global_dt_ / (double) (1 << L);
		int32_t *list      = Ls_.clu[L];
		const int counterL = acti_counter_[L];
		const int gf       = grid_for((long long) n * (NC + 1));
		ensure_scratch(n);  // a growth of the pool releases the list scratch; the reassignment uses its marks
		epoch_ += 2;
		run_k(DG_K_REGRID, n, [&] {
			k_regrid<M><<<gf, BLOCK, 0, st_>>>(P_, C_, Ls_.split, list, n, L, counterL, Ls_.fresh, epoch_ - 1, d_cnt_);
		});
		const bool ordered = opts_ & DG_OPT_ORDERED_LISTS;
		run_k(DG_K_REASSIGN, n, [&] {
			k_repair<M><<<gf, BLOCK, 0, st_>>>(P_, C_, Ls_.fresh, list, n, L, dtL, counterL, Ls_, d_cnt_, ordered ? stay_marks() : nullptr);
			// the cells that stay at level L, in their list order (the count goes to n_tmp, which the
			// reassignment of the new cells then appends to)
			if (ordered) {
				size_t bytes = sel_tmp_bytes_;
				DG_CUDA(cub::DeviceSelect::Flagged(stay_marks() + stay_bytes(scratch_cap_), bytes, list, stay_marks(),
				                                   Ls_.tmp, &d_cnt_->n_tmp, n, st_));
			}
		});
		run_k(DG_K_REASSIGN, 0, [&] { k_reassign_fresh<M><<<grid_for(n), BLOCK, 0, st_>>>(P_, C_, L, dtL, counterL, Ls_, d_cnt_); });
		std::swap(Ls_.clu[L], Ls_.tmp);
		DG_CUDA(cudaGetLastError());
	}

	void flush(int L) {
		if (h_cnt_->buf[L] == 0) return;
		run_k(DG_K_FLUSH, h_cnt_->buf[L], [&] {
			k_flush<<<grid_for(h_cnt_->buf[L]), BLOCK, 0, st_>>>(P_, Ls_.buf[L], &d_cnt_->buf[L], Ls_.clu[L],
			                                                   &d_cnt_->clu[L], L, d_cnt_);
		});
		DG_CUDA(cudaMemsetAsync(&d_cnt_->buf[L], 0, sizeof(int), st_));
		DG_CUDA(cudaGetLastError());
	}

	// The end of a substep that the host ran (impl/integrate.hpp:56-67). Returns whether a NaN ends the step.
	bool substep_end(int L) {
		acti_counter_[L] = (acti_counter_[L] + 1) % 2;
		acti_time_[L] += global_dt_ / (double) (1 << L);
		flush(L);
		sync_counters();
		check_status();
		n_split_total_ += h_cnt_->n_split;
		n_unsplit_total_ += h_cnt_->n_unsplit;
		n_substeps_++;
		updates_ += h_cnt_->clu[L];
		return h_cnt_->status & ST_NAN;
	}

	// The next substep of the global step (impl/integrate.hpp:25-39): sequence value `seq` and the next level
	// index `l` to look at in it (MAX_ACTI: the next value is due). Returns the level, -1 at the step's end.
	int next_substep(int &seq, int &l) {
		while (true) {
			if (l >= MAX_ACTI) {
				int finest = max_acti_;
				for (int k = MAX_ACTI - 1; k > finest; --k)
					if (h_cnt_->clu[k] > 0) {
						finest = k;
						break;
					}
				const int stride = 1 << (MAX_ACTI - 1 - finest);
				seq              = (seq / stride + 1) * stride;
				if (seq > 1 << (MAX_ACTI - 1)) return -1;
				l = 0;
			}
			while (l < MAX_ACTI) {
				const int k = l++;
				if (seq % (1 << k) != 0) continue;
				const int L = MAX_ACTI - k - 1;
				if (h_cnt_->clu[L] > 0 && L > max_acti_) {
					max_acti_     = L;
					acti_time_[L] = acti_time_[L - 1];
				}
				if (L <= max_acti_) return L;
			}
		}
	}

	// ---- device-resident runs (run.cuh) ---------------------------------------------------------

	// Largest cluster a run takes. Above it a substep's launches fill the GPU, and each of them has the
	// registers and block size of its own stage, where a run has one for all. With the limit between 32768 and 98304
	// cells steps take the same (a 32x16x16 + 3-level shock-drop, clusters of 17 thousand cells on average, 137 to 133 ms
	// for two steps; 64x16x16 + 4 levels 664 to 675 for one); with 16384 a 128x64 + 5-level cylinder loses, 109 ms against 80.
	static constexpr int RUN_CELLS = 1 << 16;
	// Largest cluster for which a run is one thread-block cluster (its barrier is 0.35 us, the grid's 1.3):
	// up to about here the run of sixteen SMs is as fast as the one of all (three steps of a 64x32 + 3-level shock-drop
	// 107 ms against 118, twelve of a 16^2 + 2-level quadrant problem 23 against 27).
	static constexpr int RUN_CLUSTER_CELLS = 2048;
	// Solvers side by side from which each takes one thread-block cluster, whatever its size.
	static constexpr int RUN_PEERS = 9;

	template<bool V, class S>
	void launch_run(const RunArgs &a, bool clustered) {
		auto *fn = k_run<M, V, S>;
		cudaLaunchConfig_t cfg{};
		cudaLaunchAttribute at[1];
		cfg.blockDim = RUN_THREADS;
		cfg.stream   = st_;
		cfg.attrs    = at;
		cfg.numAttrs = 1;
		if (clustered) {
			DG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
			if (run_cluster_ == 0) {
				// sixteen blocks where the device can place such a cluster, else the portable eight
				at[0].id               = cudaLaunchAttributeClusterDimension;
				at[0].val.clusterDim.x = 16;
				at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
				cfg.gridDim            = 16;
				int fit                = 0;
				if (cudaOccupancyMaxActiveClusters(&fit, fn, &cfg) != cudaSuccess) {
					cudaGetLastError();
					fit = 0;
				}
				run_cluster_ = fit > 0 ? 16 : 8;
			}
			at[0].id               = cudaLaunchAttributeClusterDimension;
			at[0].val.clusterDim.x = run_cluster_;
			at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
			cfg.gridDim            = run_cluster_;
		} else {
			int dev = 0, sms = 0;
			DG_CUDA(cudaGetDevice(&dev));
			DG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
			at[0].id              = cudaLaunchAttributeCooperative;
			at[0].val.cooperative = 1;
			cfg.gridDim           = sms;
		}
		DG_CUDA(cudaLaunchKernelEx(&cfg, fn, a));
		n_launches_++;
	}

	// The largest cluster of up to `limit` cells.
	long long most_cells(int limit) const {
		long long most = 0;
		for (int l = 0; l < MAX_ACTI; ++l)
			if (h_cnt_->clu[l] <= limit) most = std::max<long long>(most, h_cnt_->clu[l]);
		return most;
	}

	// Starts a run of the substeps from (seq, l) on, which lasts until the global step is done or the host is
	// needed; clusters above `limit` cells are left to the host.
	void run_begin(int seq, int l, int limit, bool clustered) {
		static_assert(sizeof(RunArgs) <= 4096 && sizeof(Counters) % 4 == 0, "a run's arguments are kernel parameters");
		const long long most = most_cells(limit);
		ensure_scratch(std::min<long long>(std::max<long long>(most + most / 2, 4096), limit));
		RunArgs a{};
		a.P            = P_;
		a.C            = C_;
		a.B            = B_;
		a.Ls           = Ls_;
		a.cnt          = d_cnt_;
		a.in.sch       = {max_acti_, stamp_, epoch_, 0, {}, {}};
		a.in.seq       = seq;
		a.in.l         = l;
		std::copy(acti_counter_, acti_counter_ + MAX_ACTI, a.in.sch.counter);
		std::copy(acti_time_, acti_time_ + MAX_ACTI, a.in.sch.time);
		a.out       = h_run_;
		a.out_cnt   = h_cnt_;
		a.bar       = d_bar_;
		a.global_dt = global_dt_;
		a.limiter   = limiter_;
		a.sigma     = sigma_ ? 1 : 0;
		a.rows      = (int) std::min<long long>(scratch_cap_, limit);
		a.clustered = clustered ? 1 : 0;
		h_run_->stop = -1;
		if (!clustered) DG_CUDA(cudaMemsetAsync(d_bar_, 0, sizeof(unsigned), st_));
		if constexpr (!M::VISC) {
			if (mixed_) launch_run<false, float>(a, clustered);
			else launch_run<false, double>(a, clustered);
		} else if constexpr (!M::MULTI) {
			if (mixed_) launch_run<true, float>(a, clustered);
			else launch_run<true, double>(a, clustered);
		} else {
			if (visc_ && mixed_) launch_run<true, float>(a, clustered);
			else if (visc_) launch_run<true, double>(a, clustered);
			else if (mixed_) launch_run<false, float>(a, clustered);
			else launch_run<false, double>(a, clustered);
		}
	}

	// Waits for the run. The host's schedule state, lists and counters are current afterwards. Returns why the
	// run ended (RunStop); `L` is the level of an unfinished substep.
	int run_end(int &seq, int &l, int &L) {
		lost = true;  // the lists are in the run's hands until its state is here
		DG_CUDA(cudaStreamSynchronize(st_));
		const RunState &h = *h_run_;
		if (h.stop < 0) throw dg_error(DG_ERR_CUDA, "a grid barrier of a device-resident run gave up waiting");
		lost      = false;
		max_acti_ = h.sch.max_acti;
		stamp_    = h.sch.stamp;
		epoch_    = h.sch.epoch;
		std::copy(h.sch.counter, h.sch.counter + MAX_ACTI, acti_counter_);
		std::copy(h.sch.time, h.sch.time + MAX_ACTI, acti_time_);
		seq = h.seq;
		l   = h.l;
		L   = h.L;
		std::copy(h.clu, h.clu + MAX_ACTI, Ls_.clu);
		Ls_.tmp = h.tmp;
		n_split_total_ += h.splits;
		n_unsplit_total_ += h.unsplits;
		updates_ += h.updates;
		n_substeps_ += h.substeps;
		return h.stop;
	}

	// A global step of this solver in the making: runs on the device, and what a run leaves to the host.
	struct Step {
		int seq = 0, l = MAX_ACTI;
		bool broke = false, done = false;
		long long runs = 0, stops = 0, by_host = 0;
	};
	void begin_step(int signal) {
		need_state();
		C_.signal  = signal;
		C_.coarsen = (n_global_ % coarsen_every_) == 0;
	}
	// Up to the next run: substeps of clusters above `limit` are the host's. False when the step is over.
	bool run_due(Step &p, int limit) {
		while (!p.broke && !p.done) {
			int s = p.seq, k = p.l;
			const int next = next_substep(s, k);
			if (next < 0) {
				p.done = true;
			} else if (h_cnt_->clu[next] <= limit) {
				return true;
			} else {
				p.seq = s;
				p.l   = k;
				host_substep(next);
				p.broke = substep_end(next);
				++p.by_host;
			}
		}
		return false;
	}
	// The same, and starts the run.
	bool advance(Step &p, int limit, bool clustered) {
		if (!run_due(p, limit)) return false;
		run_begin(p.seq, p.l, limit, clustered);
		++p.runs;
		return true;
	}
	// The substep that a run which ended for `stop` left to the host; `L` is its level.
	void after_run(Step &p, int stop, int L) {
		p.done = stop == RUN_DONE;
		if (stop == RUN_STATUS) {
			check_status();
			p.broke = h_cnt_->status & ST_NAN;
		} else if (stop == RUN_CAPACITY) {
			// the run closed before the regrid of substep L
			check_status();
			const int n = h_cnt_->clu[L];
			epoch_ += EPOCH_EST<M>;
			grow_for_splits();
			substep_tail(L, n);
			p.broke = substep_end(L);
			++p.stops;
			++p.by_host;
		} else if (stop == RUN_LARGE) {
			++p.stops;
		}
	}
	// The end of a run, and of the substep that it left to the host.
	void settle(Step &p) {
		int L          = 0;
		const int stop = run_end(p.seq, p.l, L);
		after_run(p, stop, L);
	}
	void host_substep(int L) {
		const int n = h_cnt_->clu[L];
		substep_head(L);
		substep_tail(L, n);
	}
	// Garbage collection and the re-sort after a complete global step; the stream may still be at work.
	void finish_step() {
		n_global_++;
		if (gc_due()) gc();
		if (resort_) resort();
	}

public:
	// Integrator::integrate (impl/integrate.hpp:12-87)
	void step(int signal, int *force_break, double *global_dt, dg_substep_fn fn, void *user, int peers = 1) override {
		begin_step(signal);
		*force_break = 0;
		*global_dt   = global_dt_;
		Step p;
		// Runs on the device serve the default stage choices; the host issues a substep's stages one by one
		// where a callback or the timing of every stage asks for it, and for clusters that fill the GPU.
		if (!fn && !prof_ && opts_ == DG_OPT_DEFAULT) {
			while (run_due(p, RUN_CELLS)) {
				const bool clustered = peers >= RUN_PEERS || most_cells(RUN_CELLS) <= RUN_CLUSTER_CELLS;
				int stop, L;
				{
					// a grid-wide run takes every SM; two of them wait for one another on the host, not on the GPU.
					// What the host does for a solver goes on beside another's run
					std::unique_lock<std::mutex> hold(whole_gpu(), std::defer_lock);
					if (!clustered) hold.lock();
					advance(p, RUN_CELLS, clustered);
					stop = run_end(p.seq, p.l, L);
				}
				after_run(p, stop, L);
			}
		} else {
			for (int L; !p.broke && (L = next_substep(p.seq, p.l)) >= 0;) {
				host_substep(L);
				p.broke = substep_end(L);
				if (!p.broke && fn)
					fn(user, L, acti_time_[L], (int) n_substeps_, global_dt_ / (double) (1 << L), h_cnt_->clu[L]);
			}
		}
		if (p.broke) {
			*force_break = 1;
			return;
		}
		finish_step();
		DG_CUDA(cudaStreamSynchronize(st_));
		drain_events();
	}

	void set_resort(bool on) { resort_ = on; }

	// Morton re-sort of the node pool by (cluster, Z-order) at the end of a global step, when every
	// ACTI buffer is empty: each cluster becomes one contiguous slot range and its list the identity
	// over that range.
	void resort() {
		for (int l = 0; l < MAX_ACTI; ++l)
			if (h_cnt_->buf[l] != 0) return;
		const int top = h_cnt_->top;
		const int n   = top - 1;
		if (n <= 0) return;
		ensure_spare();
		const int top_level = std::min(max_tree_level_, SORT_LEVELS<D>);
		int bits            = D * top_level;
		while (bits < 31 && (1 << bits) <= top) ++bits;
		const int end_bit = bits + SORT_CODE_BITS;
		static_assert(D * SORT_LEVELS<D> + SORT_CODE_BITS <= 64, "a sort key has 64 bits");
		size_t temp = 0;
		DG_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, temp, (uint64_t *) nullptr, (uint64_t *) nullptr,
		                                        (int32_t *) nullptr, (int32_t *) nullptr, n, 0, end_bit, st_));
		const size_t need = align_up(sizeof(uint64_t) * n) * 2 + align_up(sizeof(int32_t) * n) * 2 +
		                    align_up(sizeof(int32_t) * (top + 1)) + align_up(temp);
		if (need > sort_bytes_) {
			mem_free(sort_mem_, st_);
			sort_mem_   = nullptr;
			sort_bytes_ = 0;
			// half as much again for a tree that grows, where there is room for it
			size_t got    = need + need / 2;
			cudaError_t e = mem_alloc(&sort_mem_, got, st_);
			if (e == cudaErrorMemoryAllocation) {
				cudaGetLastError();
				got = need;
				e   = mem_alloc(&sort_mem_, got, st_);
			}
			if (e != cudaSuccess) sort_mem_ = nullptr;
			DG_CUDA(e);
			sort_bytes_ = got;
		}
		char *b          = (char *) sort_mem_;
		uint64_t *k_in   = (uint64_t *) b;
		b += align_up(sizeof(uint64_t) * n);
		uint64_t *k_out = (uint64_t *) b;
		b += align_up(sizeof(uint64_t) * n);
		int32_t *v_in = (int32_t *) b;
		b += align_up(sizeof(int32_t) * n);
		int32_t *v_out = (int32_t *) b;
		b += align_up(sizeof(int32_t) * n);
		int32_t *newidx = (int32_t *) b;
		b += align_up(sizeof(int32_t) * (top + 1));
		void *tmp = b;
		const int g = grid_for(n);
		run_k(DG_K_OTHER, 0, [&] { k_sort_keys<D><<<g, BLOCK, 0, st_>>>(P_, top, top_level, bits, k_in, v_in); });
		DG_CUDA(cub::DeviceRadixSort::SortPairs(tmp, temp, k_in, k_out, v_in, v_out, n, 0, end_bit, st_));
		run_k(DG_K_OTHER, 0, [&] { k_sort_inverse<<<g, BLOCK, 0, st_>>>(v_out, n, newidx); });
		auto rows = [&](const RowTable &t) {
			run_k(DG_K_OTHER, 0, [&] { k_rows<<<dim3(grid_for(top, 148 * 4), t.n), BLOCK, 0, st_>>>(t, top, v_out, newidx); });
		};
		auto words = [&](const Field &f, const void *src, void *dst) {
			run_k(DG_K_OTHER, 0, [&] {
				k_row_words<<<grid_for((long long) top * (f.elem / 8)), BLOCK, 0, st_>>>((const double *) src, (double *) dst,
				                                                                        (int) (f.elem / 8), top, v_out);
			});
		};
		auto fo = fields(P_);
		if (second_pool()) {
			if (spare_dirty_) DG_CUDA(cudaMemsetAsync(spare_mem_, 0, pool_bytes(P_), st_));
			spare_dirty_ = false;
			Pool NP      = P_;
			place_fields(NP, spare_mem_);
			auto fn = fields(NP);
			RowTable t{};
			for (size_t k = 0; k < fo.size(); ++k) {
				if (fo[k].comps <= 0 || fo[k].stay) continue;
				if (fo[k].elem > 8) words(fo[k], *fo[k].ptr, *fn[k].ptr);
				else add_rows(t, fo[k], *fo[k].ptr, P_.cap, *fn[k].ptr, P_.cap, true);
			}
			rows(t);
			std::swap(pool_mem_, spare_mem_);
			spare_bytes_ = pool_bytes(P_);
			P_           = NP;
		} else {
			// each field in turn: permuted into the spare buffer, then copied back over slots [1, top)
			for (size_t k = 0; k < fo.size(); ++k) {
				const int comps   = fo[k].comps;
				const size_t elem = fo[k].elem;
				if (comps <= 0 || fo[k].stay) continue;
				if (elem > 8) {
					words(fo[k], *fo[k].ptr, spare_mem_);
				} else {
					RowTable t{};
					add_rows(t, fo[k], *fo[k].ptr, P_.cap, spare_mem_, P_.cap, true);
					rows(t);
				}
				DG_CUDA(cudaMemcpy2DAsync((char *) *fo[k].ptr + elem, elem * (size_t) P_.cap, (const char *) spare_mem_ + elem,
				                          elem * (size_t) P_.cap, elem * (size_t) n, comps, cudaMemcpyDeviceToDevice, st_));
			}
		}
		LevelRanges r{};
		int most   = 0;
		r.first[0] = 1;
		for (int l = 0; l < MAX_ACTI; ++l) {
			r.list[l]      = Ls_.clu[l];
			r.first[l + 1] = r.first[l] + h_cnt_->clu[l];
			most           = std::max(most, h_cnt_->clu[l]);
		}
		run_k(DG_K_OTHER, 0, [&] { k_fill_ranges<<<dim3(grid_for(most), MAX_ACTI), BLOCK, 0, st_>>>(r); });
		DG_CUDA(cudaGetLastError());
	}

private:
	// Integrator::gc (impl/acti_utils.hpp:59-74): compact the node slots, then reassign every active
	// leaf to an ACTI level from its stored max_dt, resetting the hysteresis.
	void gc() {
		const int top = h_cnt_->top;
		for (int l = 0; l < MAX_ACTI; ++l)
			if (h_cnt_->buf[l] != 0) throw dg_error(DG_ERR_UNSUPPORTED, "garbage collection with non-empty ACTI buffers");
		int32_t *keep = nullptr, *newidx = nullptr;
		DG_CUDA(mem_alloc((void **) &keep, sizeof(int32_t) * (top + 1), st_));
		DG_CUDA(mem_alloc((void **) &newidx, sizeof(int32_t) * (top + 1), st_));
		const int g = grid_for(top);
		k_gc_keep<<<g, BLOCK, 0, st_>>>(P_, top, keep);
		size_t tmp_bytes = 0;
		DG_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, keep, newidx, top + 1, st_));
		void *tmp = nullptr;
		DG_CUDA(mem_alloc((void **) &tmp, tmp_bytes, st_));
		DG_CUDA(cudaMemsetAsync(keep + top, 0, sizeof(int32_t), st_));
		DG_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, keep, newidx, top + 1, st_));
		int new_top = 0;
		DG_CUDA(cudaMemcpyAsync(&new_top, newidx + top, sizeof(int), cudaMemcpyDeviceToHost, st_));
		// each field in turn: kept slots compacted into the zeroed spare buffer, which is then copied back
		// whole (slots from new_top on end up zero)
		ensure_spare();
		spare_dirty_ = true;
		auto fo = fields(P_);
		for (size_t k = 0; k < fo.size(); ++k) {
			if (fo[k].comps <= 0) continue;
			const size_t bytes = fo[k].elem * (size_t) P_.cap * fo[k].comps;
			DG_CUDA(cudaMemsetAsync(spare_mem_, 0, bytes, st_));
			k_gc_move<<<g, BLOCK, 0, st_>>>((const char *) *fo[k].ptr, (char *) spare_mem_, (int) fo[k].elem, fo[k].comps,
			                                 P_.cap, top, keep, newidx);
			DG_CUDA(cudaMemcpyAsync(*fo[k].ptr, spare_mem_, bytes, cudaMemcpyDeviceToDevice, st_));
		}
		DG_CUDA(cudaStreamSynchronize(st_));
		k_gc_remap<D><<<grid_for(new_top), BLOCK, 0, st_>>>(P_, new_top, keep, newidx);
		// full ACTI reassignment
		Counters z{};
		z.top    = new_top;
		z.status = 0;
		z.coarsest = h_cnt_->coarsest;
		// the running totals that a batched step keeps on the device carry over (the host copy is current:
		// gc runs after the step's last read-back)
		z.n_split_total    = h_cnt_->n_split_total;
		z.n_unsplit_total  = h_cnt_->n_unsplit_total;
		z.n_updates_total  = h_cnt_->n_updates_total;
		z.n_substeps_total = h_cnt_->n_substeps_total;
		DG_CUDA(cudaMemcpyAsync(d_cnt_, &z, sizeof(Counters), cudaMemcpyHostToDevice, st_));
		k_collect_active_leaves<<<grid_for(new_top), BLOCK, 0, st_>>>(P_, new_top, Ls_.fresh, &d_cnt_->n_new);
		DG_CUDA(cudaStreamSynchronize(st_));
		int n_leaves = 0;
		DG_CUDA(cudaMemcpy(&n_leaves, &d_cnt_->n_new, sizeof(int), cudaMemcpyDeviceToHost));
		k_assign<M><<<grid_for(n_leaves), BLOCK, 0, st_>>>(P_, C_, Ls_.fresh, n_leaves, global_dt_, Ls_, d_cnt_);
		DG_CUDA(cudaGetLastError());
		sync_counters();
		check_status();
		mem_free(tmp, st_);
		mem_free(keep, st_);
		mem_free(newidx, st_);
		n_gc_++;
	}

public:
	long long cell_count() override {
		long long n = 0;
		for (int l = 0; l < MAX_ACTI; ++l) n += h_cnt_->clu[l] + h_cnt_->buf[l];
		return n;
	}

	long long read_fields(const dg_cell_fields &f, long long max_cells) override {
		const long long n = cell_count();
		if (n > max_cells) throw dg_error(DG_ERR_ARG, "read buffer too small");
		if (n == 0) return 0;
		// one buffer, the arrays one after another
		struct Part {
			void *host;
			size_t bytes;
		};
		const size_t d = sizeof(double) * (size_t) n, w = sizeof(int32_t) * (size_t) n;
		const Part part[10] = {{f.center, d * D}, {f.t, d}, {f.u, d * E}, {f.p, d * E}, {f.error, d}, {f.max_dt, d}, {f.cfl, d},
		                       {f.k, d * M::P}, {f.level, w}, {f.acti, w}};
		size_t at[10], total = 0;
		for (int k = 0; k < 10; ++k) at[k] = total, total += align_up(part[k].bytes);
		char *buf = nullptr;
		DG_CUDA(mem_alloc((void **) &buf, total, st_));
		const FieldArrays o{(int32_t *) (buf + at[8]), (int32_t *) (buf + at[9]), (double *) (buf + at[0]), (double *) (buf + at[1]),
		                    (double *) (buf + at[2]), (double *) (buf + at[3]), (double *) (buf + at[4]), (double *) (buf + at[5]),
		                    (double *) (buf + at[6]), (double *) (buf + at[7])};
		long long base = 0;
		for (int pass = 0; pass < 2; ++pass) {
			for (int l = 0; l < MAX_ACTI; ++l) {
				const int cnt = pass == 0 ? h_cnt_->clu[l] : h_cnt_->buf[l];
				if (cnt == 0) continue;
				k_gather_fields<M><<<grid_for(cnt), BLOCK, 0, st_>>>(P_, pass == 0 ? Ls_.clu[l] : Ls_.buf[l], cnt, (int) base, o);
				base += cnt;
			}
		}
		cudaError_t e = cudaGetLastError();
		for (int k = 0; k < 10 && e == cudaSuccess; ++k)
			if (part[k].bytes > 0) e = cudaMemcpyAsync(part[k].host, buf + at[k], part[k].bytes, cudaMemcpyDeviceToHost, st_);
		if (e == cudaSuccess) e = cudaStreamSynchronize(st_);
		mem_free(buf, st_);
		if (e != cudaSuccess) throw dg_error(DG_ERR_CUDA, std::string("read_fields: ") + cudaGetErrorString(e));
		return n;
	}

	long long read_cells(int *levels, double *data, long long max_cells) override {
		constexpr int W = D + 1 + 2 * E + 3 + M::P;
		long long n = cell_count();
		if (n > max_cells) throw dg_error(DG_ERR_ARG, "read buffer too small");
		if (n > read_cap_) {
			mem_free(d_read_, st_);
			mem_free(d_readlv_, st_);
			DG_CUDA(mem_alloc((void **) &d_read_, sizeof(double) * W * n, st_));
			DG_CUDA(mem_alloc((void **) &d_readlv_, sizeof(int32_t) * 2 * n, st_));
			read_cap_ = n;
		}
		long long base = 0;
		for (int pass = 0; pass < 2; ++pass) {
			for (int l = 0; l < MAX_ACTI; ++l) {
				int cnt = pass == 0 ? h_cnt_->clu[l] : h_cnt_->buf[l];
				if (cnt == 0) continue;
				const int32_t *list = pass == 0 ? Ls_.clu[l] : Ls_.buf[l];
				k_gather_cells<M><<<grid_for(cnt), BLOCK, 0, st_>>>(P_, list, cnt, (int) base, d_read_, d_readlv_);
				base += cnt;
			}
		}
		DG_CUDA(cudaGetLastError());
		DG_CUDA(cudaMemcpyAsync(data, d_read_, sizeof(double) * W * n, cudaMemcpyDeviceToHost, st_));
		DG_CUDA(cudaMemcpyAsync(levels, d_readlv_, sizeof(int32_t) * 2 * n, cudaMemcpyDeviceToHost, st_));
		DG_CUDA(cudaStreamSynchronize(st_));
		return n;
	}

	// `width` doubles per active cell, gathered by `launch(list, count, base, out)` in read_cells' order.
	template<class F>
	long long read_per_cell(double *data, long long max_cells, int width, const char *what, F launch) {
		const long long n = cell_count();
		if (n > max_cells) throw dg_error(DG_ERR_ARG, "read buffer too small");
		double *d_out = nullptr;
		DG_CUDA(mem_alloc((void **) &d_out, sizeof(double) * width * (n > 0 ? n : 1), st_));
		long long base = 0;
		for (int pass = 0; pass < 2; ++pass) {
			for (int l = 0; l < MAX_ACTI; ++l) {
				const int cnt = pass == 0 ? h_cnt_->clu[l] : h_cnt_->buf[l];
				if (cnt == 0) continue;
				launch(pass == 0 ? Ls_.clu[l] : Ls_.buf[l], cnt, (int) base, d_out);
				base += cnt;
			}
		}
		cudaError_t e = cudaGetLastError();
		if (e == cudaSuccess && n > 0) e = cudaMemcpyAsync(data, d_out, sizeof(double) * width * n, cudaMemcpyDeviceToHost, st_);
		if (e == cudaSuccess) e = cudaStreamSynchronize(st_);
		mem_free(d_out, st_);
		if (e != cudaSuccess) throw dg_error(DG_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
		return n;
	}

	// Limited slopes of the active cells, [D][E] per cell, in read_cells' order.
	long long read_slopes(double *data, long long max_cells) override {
		return read_per_cell(data, max_cells, D * E, "read_slopes", [&](const int32_t *list, int cnt, int base, double *o) {
			k_gather_slopes<M><<<grid_for(cnt), BLOCK, 0, st_>>>(P_, list, cnt, base, o);
		});
	}

	// Regrid-forecaster features, [5 + 5D] per active cell, in read_cells' order.
	long long forecast_features(double *data, long long max_cells) override {
		return read_per_cell(data, max_cells, 5 + 5 * D, "forecast_features",
		                     [&](const int32_t *list, int cnt, int base, double *o) {
			                     k_forecast_features<M><<<grid_for(cnt), BLOCK, 0, st_>>>(P_, C_, list, cnt, base, o);
		                     });
	}
	int dims() const override { return D; }

	long long tree_size() override { return h_cnt_->top; }

	// The whole node pool, slots [0, top), component-major as the pool stores it: parent[n],
	// child[C][n], level[n], flags[n], p[E][n], meta[4][n] = {acti_level, error, max_dt, cfl}. Internal,
	// inactive and garbage slots included: what a hyper-tree writer walks from the root.
	long long read_tree(int32_t *parent, int32_t *child, int32_t *level, uint32_t *flags, double *p, double *meta,
	                    long long max_nodes) override {
		const long long n = h_cnt_->top;
		if (n > max_nodes) throw dg_error(DG_ERR_ARG, "read buffer too small");
		const size_t cap = (size_t) P_.cap, nn = (size_t) n;
		std::vector<int8_t> lv(nn), ac(nn);
		auto rows = [&](void *dst, const void *src, size_t elem, int comps) {
			DG_CUDA(cudaMemcpy2DAsync(dst, elem * nn, src, elem * cap, elem * nn, comps, cudaMemcpyDeviceToHost, st_));
		};
		rows(parent, P_.parent, 4, 1);
		rows(child, P_.child, 4, NC);
		rows(lv.data(), P_.level, 1, 1);
		rows(ac.data(), P_.acti, 1, 1);
		rows(flags, P_.flags, 4, 1);
		rows(p, P_.p, 8, E);
		rows(meta + nn, P_.err, 8, 1);
		rows(meta + 2 * nn, P_.maxdt, 8, 1);
		rows(meta + 3 * nn, P_.cfl, 8, 1);
		DG_CUDA(cudaStreamSynchronize(st_));
		for (size_t i = 0; i < nn; ++i) {
			level[i] = lv[i];
			meta[i]  = (double) ac[i];
			flags[i] &= F_PUBLIC;
		}
		return n;
	}

	// Forecast-driven regrid: F_HOLD on the active cells (read_cells' order) and the interval in global
	// steps between coarsening passes (1 = every step, the reference's behaviour).
	void set_hold(const uint8_t *hold, long long n) override {
		if (n != cell_count()) throw dg_error(DG_ERR_ARG, "dg_set_hold: one entry per active cell expected");
		uint8_t *d = nullptr;
		DG_CUDA(mem_alloc((void **) &d, n > 0 ? n : 1, st_));
		cudaError_t e = n > 0 ? cudaMemcpyAsync(d, hold, n, cudaMemcpyHostToDevice, st_) : cudaSuccess;
		long long base = 0;
		for (int pass = 0; e == cudaSuccess && pass < 2; ++pass) {
			for (int l = 0; l < MAX_ACTI; ++l) {
				const int cnt = pass == 0 ? h_cnt_->clu[l] : h_cnt_->buf[l];
				if (cnt == 0) continue;
				k_set_hold<M><<<grid_for(cnt), BLOCK, 0, st_>>>(P_, pass == 0 ? Ls_.clu[l] : Ls_.buf[l], cnt, (int) base, d);
				base += cnt;
			}
		}
		if (e == cudaSuccess) e = cudaGetLastError();
		if (e == cudaSuccess) e = cudaStreamSynchronize(st_);
		mem_free(d, st_);
		if (e != cudaSuccess) throw dg_error(DG_ERR_CUDA, std::string("set_hold: ") + cudaGetErrorString(e));
	}
	void set_coarsen_interval(int k) override {
		if (k < 1) throw dg_error(DG_ERR_ARG, "dg_set_coarsen_interval: interval must be >= 1");
		coarsen_every_ = k;
	}

	// Gradients of the gradient inputs, [D][G] per active cell, in read_cells' order.
	long long read_gradients(double *data, long long max_cells) override {
		if constexpr (M::G == 0) {
			throw dg_error(DG_ERR_UNSUPPORTED, "dg_read_gradients: the Euler model has no gradient inputs");
		} else {
			if (!visc_)
				throw dg_error(DG_ERR_UNSUPPORTED, "dg_read_gradients: gradients are kept only when the case has viscous "
				                                   "or heat-conduction terms");
			return read_per_cell(data, max_cells, D * M::G, "read_gradients",
			                     [&](const int32_t *list, int cnt, int base, double *o) {
				                     k_gather_grads<M><<<grid_for(cnt), BLOCK, 0, st_>>>(P_, list, cnt, base, o);
			                     });
		}
	}

	// Same records as read_cells, gathered through caller-owned device scratch of `bytes` bytes;
	// allocates nothing.
	int model_id() const override { return M::ID; }

	void prepare_noalloc() override {
		cudaFuncAttributes a{};
		DG_CUDA(cudaFuncGetAttributes(&a, k_gather_cells<M>));
	}

	long long read_cells_via(int *levels, double *data, long long max_cells, void *scratch, size_t bytes) override {
		constexpr int W = D + 1 + 2 * E + 3 + M::P;
		const long long n = cell_count();
		if (n > max_cells) throw dg_error(DG_ERR_ARG, "read buffer too small");
		const size_t rec_bytes = align_up(sizeof(double) * W * (size_t) n);
		const size_t need      = rec_bytes + sizeof(int32_t) * 2 * (size_t) n;
		const size_t per_cell  = sizeof(double) * W + sizeof(int32_t) * 2;
		if (need > bytes)
			throw dg_error(DG_ERR_CAPACITY, "dg_read_cells_noalloc: " + std::to_string(n) + " active cells need " +
			                                    std::to_string(need) + " bytes of scratch; the allocation-free scratch holds " +
			                                    std::to_string(bytes) + " bytes (about " +
			                                    std::to_string((bytes - 256) / per_cell) + " cells of this model)");
		double *d_rec = (double *) scratch;
		int32_t *d_lv = (int32_t *) ((char *) scratch + rec_bytes);
		long long base = 0;
		for (int pass = 0; pass < 2; ++pass) {
			for (int l = 0; l < MAX_ACTI; ++l) {
				int cnt = pass == 0 ? h_cnt_->clu[l] : h_cnt_->buf[l];
				if (cnt == 0) continue;
				const int32_t *list = pass == 0 ? Ls_.clu[l] : Ls_.buf[l];
				k_gather_cells<M><<<grid_for(cnt), BLOCK, 0, st_>>>(P_, list, cnt, (int) base, d_rec, d_lv);
				base += cnt;
			}
		}
		DG_CUDA(cudaGetLastError());
		if (n > 0) {
			DG_CUDA(cudaMemcpyAsync(data, d_rec, sizeof(double) * W * n, cudaMemcpyDeviceToHost, st_));
			DG_CUDA(cudaMemcpyAsync(levels, d_lv, sizeof(int32_t) * 2 * n, cudaMemcpyDeviceToHost, st_));
		}
		DG_CUDA(cudaStreamSynchronize(st_));
		return n;
	}

	void stats(dg_stats *o) override {
		std::memset(o, 0, sizeof(*o));
		for (int l = 0; l < MAX_ACTI; ++l) {
			o->n_clusters[l]   = h_cnt_->clu[l];
			o->n_buffers[l]    = h_cnt_->buf[l];
			o->acti_time[l]    = acti_time_[l];
			o->acti_counter[l] = acti_counter_[l];
		}
		o->tree_size      = h_cnt_->top + pruned_;
		o->n_splits       = n_split_total_;
		o->n_unsplits     = n_unsplit_total_;
		o->n_gc           = n_gc_;
		o->n_substeps     = n_substeps_;
		o->n_global_steps = n_global_;
		o->cell_updates   = updates_;
		o->max_acti_level = max_acti_;
		o->global_dt      = global_dt_;
		o->n_launches     = n_launches_;
		for (int k = 0; k < DG_NK; ++k) {
			o->kernel_ms[k]       = kms_[k];
			o->kernel_launches[k] = klaunch_[k];
			o->kernel_cells[k]    = kcells_[k];
		}
	}
};

SolverBase *make_solver_euler(const dg_case &c);
SolverBase *make_solver_ns(const dg_case &c);
SolverBase *make_solver_multi(const dg_case &c);
class BatchBase;
BatchBase *make_batch_euler(const std::vector<SolverBase *> &s);
BatchBase *make_batch_ns(const std::vector<SolverBase *> &s);
BatchBase *make_batch_multi(const std::vector<SolverBase *> &s);

}  // namespace dg
