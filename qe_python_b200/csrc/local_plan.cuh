// Plan object of the local H|psi> operator, shared by the generic
// (local_hpsi.cu) and the line-transform (local_lines.cuh) kernels.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

#include "qeb_common.cuh"

// k points one batched local apply handles (qeb_apply_local_multi).
#define QEB_MAX_KBATCH 16

struct qeb_local_plan {
  int nx, ny, nz;
  int64_t npw;
  int nst;       // occupied (x, y) sticks, ordered by (y, x)
  int nay;       // active y rows
  int nx_pad;    // shared-memory row stride of the active-row plane
  int ny_pad;    // shared-memory stride of the column lines
  int nz_pad;    // shared-memory stride of the stick lines
  int precision; // QEB_F64 or QEB_F32
  int device;
  qeb::FftDesc fx, fy, fz;
  // Line transforms: every axis has a two-factor split n = n1 n2
  // (line_lengths.cuh) and the plane fits shared memory; else the generic
  // kernels run.
  bool lines;
  // Static plane kernel of square planes whose sticks all lie in
  // [0, line_k n2) or [n - line_k n2, n) of x and y: the plane holds the rows
  // of those 2 line_k blocks of x.  0: run-time kernel, the blocks of the
  // masks below, also where the rows of all 2 line_k blocks exceed shared
  // memory (FP64, 192 points).  QEB_PRUNE_PLANE=0 keeps a plan on it.
  int line_k;
  int line_rows;     // rows (x values) the plane holds
  int line_columns;  // columns per batch of the run-time kernel
  // Bit i: block i of n2 consecutive values [n2 i, n2 (i + 1)) of the axis
  // holds a stick (x, y) or an entry (z); the others are zero on input and
  // unread on output.
  uint32_t xmask, ymask, zmask;
  // device arrays (plan-owned)
  int32_t* entry_g;      // npw: plane-wave row, CSR-ordered by (stick, z)
  int32_t* entry_z;      // npw: z slot
  int32_t* entry_stick;  // npw: stick index
  int32_t* stick_off;    // nst + 1
  int32_t* stick_pos;    // nst: ay * nx_pad + x (shared-memory plane position)
  int32_t* ay_to_y;      // nay
  int32_t* y_to_ay;      // ny (-1 when the row holds no stick)
  // line transforms only, else null
  int32_t* entry_pos;    // npw: (stick % 32) * (nz | 1) + z, the z pass's shared-memory position
  int32_t* stick_map;    // ny x line_rows: stick at (y, row), or -1
  void* tw;              // forward twiddles: nx, then ny, then nz entries (complex T)
};

namespace qeb {

// The factors n = n1 n2 of a line transform (false: none listed).
bool line_split(int n, int* n1, int* n2);
// Blocks the static plane kernel of n-point lines keeps at each end when every
// stick lies within `reach` values of an end, or 0 (none does).
int line_keep(int n, int reach);
// Columns per batch of the run-time plane kernel for a plan's sizes and
// line_rows; 0: the plane does not fit shared memory.
int line_columns(const qeb_local_plan* p);
// Raise the shared-memory limits of the kernels that a plan launches.
int lines_prepare(const qeb_local_plan* p);
// The three passes once for nk <= QEB_MAX_KBATCH plans on one grid (same sizes,
// precision and device): grid.z = k point; a k point gives the same bits alone
// and in a batch.  events: four, recorded around the passes, or null.
// barrier: two words of the caller's scratch for the grid barrier of the
// persistent launch (qeb_set_persistent_passes), or null.
int lines_apply(int nk, const qeb_local_plan* const* plans, void* const* sticks,
                const void* const* psi, const int64_t* ld, const int64_t* nb,
                const void* potential, const void* const* kinetic, void* const* out,
                const int64_t* ldo, cudaStream_t stream, cudaEvent_t* events,
                unsigned int* barrier);
// grid: nx ny nz doubles of scratch, or null.
int lines_density(const qeb_local_plan* p, void* sticks, double* grid, const void* psi, int64_t ld,
                  int64_t nb, const double* weights, double* density, cudaStream_t stream);

}  // namespace qeb
