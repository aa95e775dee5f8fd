// What the C entry points and batches see of a solver, and the errors it throws.
#pragma once

#include "../../include/dacti_gpu.h"

#include <cuda_runtime.h>

#include <cstdint>
#include <stdexcept>
#include <string>

namespace dg {

struct dg_error : std::runtime_error {
	int code;
	dg_error(int c, const std::string &m) :
	    std::runtime_error(m), code(c) {}
};

#define DG_CUDA(x)                                                                                     \
	do {                                                                                               \
		cudaError_t e_ = (x);                                                                          \
		if (e_ != cudaSuccess)                                                                         \
			throw ::dg::dg_error(DG_ERR_CUDA, std::string(#x) + ": " + cudaGetErrorString(e_));         \
	} while (0)

class SolverBase {
public:
	virtual ~SolverBase() = default;
	// `peers`: solvers that step at the same time on streams of their own (1: this one has the GPU)
	virtual void step(int signal, int *force_break, double *global_dt, dg_substep_fn fn, void *user, int peers = 1) = 0;
	virtual long long cell_count() = 0;
	virtual long long read_cells(int *levels, double *data, long long max_cells) = 0;
	virtual long long read_fields(const dg_cell_fields &f, long long max_cells) = 0;
	virtual long long read_cells_via(int *levels, double *data, long long max_cells, void *scratch, size_t bytes) = 0;
	virtual long long read_slopes(double *data, long long max_cells) = 0;
	virtual long long read_gradients(double *data, long long max_cells) = 0;
	virtual long long forecast_features(double *data, long long max_cells) = 0;
	virtual long long tree_size() = 0;
	virtual long long read_tree(int32_t *parent, int32_t *child, int32_t *level, uint32_t *flags, double *p, double *meta,
	                            long long max_nodes) = 0;
	virtual int dims() const = 0;
	virtual void set_hold(const uint8_t *hold, long long n) = 0;
	virtual void set_coarsen_interval(int k) = 0;
	virtual void stats(dg_stats *out) = 0;
	virtual void set_stream(cudaStream_t s) = 0;
	virtual void own_stream() = 0;  // give the solver a stream of its own if it runs on the legacy default
	virtual void set_profiling(bool on) = 0;
	virtual void set_form(int form) = 0;
	virtual void set_options(int opts) = 0;
	virtual void prepare_noalloc() = 0;  // loads the read-back gather kernel on the current device
	virtual int model_id() const = 0;
	std::string last_error;
	// A run that did not leave its state has been stepping this solver: its lists and schedule are unknown, and nothing
	// but the error text and the destructor may be asked for.
	bool lost = false;
	void need_state() const {
		if (lost) throw dg_error(DG_ERR_CUDA, "the solver's state was lost when a run did not finish");
	}
};

}  // namespace dg
