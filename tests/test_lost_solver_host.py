"""A solver whose run did not finish is refused by every entry point (no GPU: a stand-in behind the handle)."""
import ctypes
import os
import subprocess

from conftest import ROOT
from dacti_b200 import solver

FAKE = r"""
#include "solver_base.h"
namespace {
// counts the calls that reach it
struct Fake : dg::SolverBase {
	int calls = 0;
	long long hit() { return ++calls; }
	void step(int, int *, double *, dg_substep_fn, void *, int) override { hit(); }
	long long cell_count() override { return hit(); }
	long long read_cells(int *, double *, long long) override { return hit(); }
	long long read_fields(const dg_cell_fields &, long long) override { return hit(); }
	long long read_cells_via(int *, double *, long long, void *, size_t) override { return hit(); }
	long long read_slopes(double *, long long) override { return hit(); }
	long long read_gradients(double *, long long) override { return hit(); }
	long long forecast_features(double *, long long) override { return hit(); }
	long long tree_size() override { return hit(); }
	long long read_tree(int32_t *, int32_t *, int32_t *, uint32_t *, double *, double *, long long) override { return hit(); }
	int dims() const override { return 2; }
	void set_hold(const uint8_t *, long long) override { hit(); }
	void set_coarsen_interval(int) override { hit(); }
	void stats(dg_stats *) override { hit(); }
	void set_stream(cudaStream_t) override { hit(); }
	void own_stream() override { hit(); }
	void set_profiling(bool) override { hit(); }
	void set_form(int) override { hit(); }
	void set_options(int) override { hit(); }
	void prepare_noalloc() override { hit(); }
	int model_id() const override { return DG_EULER; }
};
Fake fake;
struct Handle {
	dg::SolverBase *impl;
	int device;
} handle{&fake, 0};
}
extern "C" void *fake_handle() { fake.lost = true; return &handle; }
extern "C" int fake_calls() { return fake.calls; }
"""


def test_every_entry_point_refuses_a_lost_solver(tmp_path):
    src, so = tmp_path / "fake.cpp", tmp_path / "fake.so"
    src.write_text(FAKE)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "dacti_b200", "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-I", os.path.join(cuda, "include"), str(src), "-o", str(so)], check=True)
    fake, lib = ctypes.CDLL(str(so)), solver.load_library()
    fake.fake_handle.restype = ctypes.c_void_p
    h = ctypes.c_void_p(fake.fake_handle())
    i, d, n = (ctypes.c_int * 8)(), (ctypes.c_double * 64)(), ctypes.c_longlong(0)
    u, b = (ctypes.c_uint * 8)(), (ctypes.c_ubyte * 8)()
    dp, ip = ctypes.cast(d, ctypes.POINTER(ctypes.c_double)), ctypes.cast(i, ctypes.POINTER(ctypes.c_int))
    f = solver.DgCellFields(ip, ip, *([dp] * 8))
    out = ctypes.c_void_p()
    calls = {
        "dg_step": lambda: lib.dg_step(h, 0, ctypes.byref(ctypes.c_int()), ctypes.byref(ctypes.c_double()), solver.SUBSTEP_FN(), None),
        "dg_step_many": lambda: lib.dg_step_many((ctypes.c_void_p * 1)(h), 1, 1, 0, (ctypes.c_int * 1)(), (ctypes.c_double * 1)(),
                                                 (ctypes.c_int * 1)()),
        "dg_batch_create": lambda: lib.dg_batch_create((ctypes.c_void_p * 1)(h), 1, ctypes.byref(out)),
        "dg_cell_count": lambda: lib.dg_cell_count(h, ctypes.byref(n)),
        "dg_read_cells": lambda: lib.dg_read_cells(h, i, d, 1, ctypes.byref(n)),
        "dg_read_cells_noalloc": lambda: lib.dg_read_cells_noalloc(h, i, d, 1, ctypes.byref(n)),
        "dg_read_fields": lambda: lib.dg_read_fields(h, ctypes.byref(f), 1, ctypes.byref(n)),
        "dg_read_slopes": lambda: lib.dg_read_slopes(h, d, 1, ctypes.byref(n)),
        "dg_read_gradients": lambda: lib.dg_read_gradients(h, d, 1, ctypes.byref(n)),
        "dg_forecast_features": lambda: lib.dg_forecast_features(h, d, 1, ctypes.byref(n)),
        "dg_tree_size": lambda: lib.dg_tree_size(h, ctypes.byref(n)),
        "dg_read_tree": lambda: lib.dg_read_tree(h, i, i, i, u, d, d, 1, ctypes.byref(n)),
        "dg_set_hold": lambda: lib.dg_set_hold(h, b, 1),
        "dg_get_stats": lambda: lib.dg_get_stats(h, ctypes.byref(solver.DgStats())),
        "dg_set_form": lambda: lib.dg_set_form(h, 0),
    }
    for name, call in calls.items():
        assert call() == -2, name
        assert b"lost" in lib.dg_last_error(h), name
    assert fake.fake_calls() == 0
