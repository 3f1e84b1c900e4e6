// kernels.h -- host-side declarations of the vfgpu kernel launchers.
#pragma once

#include <algorithm>

#include "common.cuh"
#include "ops.cuh"

namespace vfgpu {

cudaError_t apply_kernel_attributes();
TilePlan u_plan(int nx, int ny, int nz, int prec_bytes, int num_sms);
// The bounded mbarrier wait, alone: *timed_out = 1 when a
// wait on a phase that never completes (complete = 0) gave up after `cycles`.
cudaError_t wait_selftest(long long cycles, int complete, int* timed_out);

// The U operator's unit lists for one tile plan (UApplyArgs::ur): the per-(tile,
// element layer) constant-phase-field flags and the two lists built from them.
struct UnitLists {
  uint8_t* cls = nullptr;  // [ntx nty][nz - 1]; null: no lists for this plan
  int4* runs[2] = {};      // [ntx nty nz] each
  int* start[2] = {};      // [ncta0], [ncta]
  int* total = nullptr;    // [2]
  // The stencil's flags (UApplyArgs::node, srange), null where the grid or the problem takes
  // the element operator alone; cls then holds a type per (tile, plane)
  uint8_t* node = nullptr;
  int2* srange = nullptr;
};
// Device bytes of a plan's unit lists; 0 when the grid has more tile columns than the
// one-block list builder takes (its applies then split all units).
size_t unit_lists_bytes(const TilePlan& p, int nz);
UnitLists unit_lists_carve(void* base, const TilePlan& p, int nz);
// Whether the split measured faster than one wave at this plan's size in precision
// prec_bytes (8 or 4): the VFGPU_U_SPLIT_AUTO rule.
bool unit_lists_pay(const TilePlan& p, int nz, int prec_bytes);
// Rebuilds the lists from the FP64 phase field v (two launches on s).
cudaError_t build_unit_lists(const double* v, int nx, int ny, int nz, const TilePlan& p,
                             const UnitLists& L, cudaStream_t s);
// Whether the grid's U applies run in two phases (u_twophase.cuh); the scratch of one, in values,
// and the x.y partials it writes.
bool twophase_pays(int nx, int ny, int nz, int prec_bytes);
size_t twophase_scratch(int nx, int ny, int nz);
int twophase_dots(int nx, int ny, int nz);
// Whether the plan's homogeneous nodes take the stencil in precision prec_bytes: the part of the
// rule that the grid decides.  u_stencil_on adds the problem's (one material, no per-cell modulus,
// no NOCOMPRESSION); the ctx's device-buffer applies and solves follow it, the host-buffer and
// fixed-scratch applies keep the element operator.
bool stencil_pays(const TilePlan& p, int nx, int ny, int nz, int prec_bytes);
inline size_t stencil_range_bytes(const TilePlan& p) { return sizeof(int2) * (size_t)p.st.blocks(); }
// The node flags from the FP64 phase field and the Dirichlet bits; then, per plan, the
// unit lists from them (with the nodes of listed units alone handed to the elements) and the
// stencil blocks' plane ranges.  Plans of the same tiles may share the node flags.
cudaError_t build_node_flags(const double* v, const uint8_t* bc, int nx, int ny, int nz, uint8_t* node,
                             cudaStream_t s);
cudaError_t build_stencil_lists(uint8_t* node, int2* range, int nx, int ny, int nz, const TilePlan& p,
                                const UnitLists& L, cudaStream_t s);
template <typename T> void use_unit_lists(UApplyArgs<T>& A, const UnitLists& L) {
  for (int l = 0; l < 2; l++) {
    A.ur[l] = L.cls ? L.runs[l] : nullptr;
    A.ustart[l] = L.cls ? L.start[l] : nullptr;
  }
  A.utotal = L.cls ? L.total : nullptr;
  A.node = L.cls ? L.node : nullptr;
  A.srange = L.srange;
}

template <typename T>
cudaError_t launch_u_apply(const UApplyArgs<T>& A, const TilePlan& p, const LayerTable& L,
                           cudaStream_t s);
}  // namespace vfgpu
