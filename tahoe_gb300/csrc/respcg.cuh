// Resident PCG: data shared by its host planning and its kernels.
#pragma once

#include <vector>

#include "tg_internal.h"

namespace tg {

constexpr int kResChunkRows = 8;  // rows of one warp, four lanes each

constexpr int kResAux = 7;  // streams of a batch's cluster classes beside the context's own

// One group's structure on the device: the active rows (nodes with a free
// dof) of a mesh or of one RVE, their blocks in sliced-ELL order and their
// split over CTAs.
struct ResPlanDev {
  const int* act_node;    // rows: local node of every active row
  const int* blk;         // steps*32: block of the node-block CSR, -1 padding
  const int2* slot;       // steps*32: its contributions {first, count}, no contributions for padding
  const int* col;         // steps*32: active row index of the block's column
  const int* chunk_step;  // nchunks+1: first step of every chunk of 8 rows
  const int* part_chunk;  // k+1: first chunk of every CTA's part
  const int4* part_win;   // k: {first column, columns, first and last part whose windows hold this part's rows}
  const int* contrib;     // contribution codes of the CSR
  int rows, k, nchunks;
};

// One solve of a launch: a plan applied at an instance's offsets to one of the
// call's right-hand sides.
struct ResItem {
  int plan, seg, node_off, elem_off, vec, pad;
  long long ll;  // grid form: first word of its exchange area
};

// What one solve reports.
struct ResOut {
  double rr, rr0, unscale;
  int done, fail, iters, pad;
};

// Rows of a mesh or RVE in the kernel's order (host).
struct ResRows {
  int rows = 0;
  std::vector<int> act_node, blk, col, chunk_step, chunk_lo, chunk_hi;
};

// What a CTA and the chip hold: dynamic shared memory, the largest cluster, and
// for every cluster size the largest with as many at a time.
struct ResLimits {
  size_t smem = 0;
  int cluster = 1;
  int widest[17] = {};
};

// A split of them over CTAs for one precision (host) and its device copy.
struct ResPlan {
  int rows = 0, nchunks = 0, k = 0, warps = 0;  // warps: of every CTA
  size_t smem = 0;                              // the largest part's bytes
  bool grid = false;
  bool one = false;                             // no warp has more than one chunk
  std::vector<int> part_chunk;
  std::vector<int4> part_win;
  ResPlanDev dev{};
  int elem0 = 0;        // element that its contribution map counts from
};

// The plans of the current mesh for one precision, for a solve of the whole
// mesh or of its RVEs.
struct ResMode {
  int state = 0;  // 0 not planned, 1 resident, 2 hybrid, -1 neither
  std::vector<ResPlan> plans;
  std::vector<int> plan_of;  // plan of every RVE (one entry for a whole mesh), -1: streamed
  int streamed = 0;          // RVEs that do not fit
  ResPlanDev* d_plans = nullptr;
  std::vector<void*> bufs;   // its device buffers
};
// Everything the resident PCG keeps with a context: device buffers go with the
// mesh, streams and events with the context.
struct ResState {
  ResMode mode[2][2];  // [precision][batch]
  ResItem* d_items = nullptr;
  ResOut* d_out = nullptr;
  int items_cap = 0;
  uint4* d_ll = nullptr;
  long long ll_cap = 0;
  cudaStream_t aux[kResAux] = {};
  cudaEvent_t fork = nullptr, join[kResAux] = {};
  bool limits_known[2] = {false, false};
  ResLimits limits[2];
};

void resident_rows(int n0, int n1, const int* rowptr, const int* col, const uint8_t* mask, ResRows& R);
bool resident_plan(const ResRows& R, int elem, int num_sms, const ResLimits& L, bool alone, ResPlan& P);

// The device copy of a template's rows and its plan for one precision
// (compose.cu), built on first use.
int template_resident(Context* c, int tpl, int precision, ResPlan& P, bool& fits);
// Appends the device form of rows / a split to a host image of ints; the
// pointers are filled once the image is on the device.
struct ResImage {
  std::vector<int> data;
  size_t rows_at(const ResRows& R);
  size_t split_at(const ResPlan& P);
};
void resident_bind_rows(ResPlanDev& D, const int* base, size_t at, const ResRows& R);
void resident_bind_split(ResPlanDev& D, const int* base, size_t at, const ResPlan& P);
int resident_slots(Context* c, long long n, const int* d_blk, const int* d_cptr, int2* d_slot);
int resident_limits(Context* c, int precision, ResLimits* limits);

}  // namespace tg
