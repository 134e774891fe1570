// Internal declarations of the B200 hot-path library (not part of the ABI).
#pragma once
#include <vector>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>

#include "../../include/ovs.h"

#define OVS_MAX_DEG 128        // longest CSR row supported (27*nshl hex bound = 216 not needed)
#define OVS_MAX_KSPACE 400     // largest Krylov space
// rows per tile of the tet edge pass: one round of its diagonal blocks, and about
// two rounds of its edges.  FP64 NS+VOF rows at 128^3 x6 with tiles of 8, 16, 32:
// 6.73, 5.91, 6.29 ms (T 0.66, 0.66, 0.81), FP32 3.72, 3.35, 3.34 (T 0.49, 0.48,
// 0.46); 48x48x96 0.733, 0.655, 0.704 and 0.407, 0.374, 0.387; tiles of 64 rows
// 0.818 and 0.459
#define OVS_TILE_ROWS 16
#define OVS_ASYNC_SLOTS 16     // assembly passes ovs_assemble_async queues before a wait
#define OVS_RED_BLOCKS 592     // fixed grid of every deterministic reduction (4 x 148 SMs)
#define OVS_RED_THREADS 256
#define OVS_COOP_MAX_BLOCKS 4096  // largest cooperative grid of the Arnoldi kernel

#define OVS_CUDA_TRY(expr)                                   \
  do {                                                       \
    cudaError_t _e = (expr);                                 \
    if (_e != cudaSuccess) {                                 \
      ovs_set_last_cuda_error(_e, #expr, __FILE__, __LINE__); \
      return OVS_ERR_CUDA;                                   \
    }                                                        \
  } while (0)

void ovs_set_last_cuda_error(cudaError_t e, const char* what, const char* file,
                             int line);

// number of field components per node of each system
static inline int ovs_sys_nf(int sys) {
  return sys == OVS_SYS_NS ? 4 : (sys == OVS_SYS_NSVOF ? 5 : 1);
}
// matrix values stored per CSR slot
static inline int ovs_sys_nv(int sys) {
  return sys == OVS_SYS_NS ? 16 : (sys == OVS_SYS_NSVOF ? 24 : 1);
}

// Device-side GMRES bookkeeping (one per context, FP64 throughout).
struct GmresDev {
  double beta;        // result of the latest Gram-Schmidt dot
  double epsnrm;      // tol * |P^-1 b|
  double unorm0;      // |P^-1 b|
  double ercheck;
  int iks;            // iterations completed
  int done;           // the step that ended the cycle (converged, breakdown or kspace), -1: a zero start; 0: running
  int breakdown;
  int converged;
  int kspace, kmin;
  int counter;        // last-block-done counter of the reductions
  int pad;
  double H[(OVS_MAX_KSPACE + 1) * OVS_MAX_KSPACE];  // column-major (kspace+1) x kspace
  double e[OVS_MAX_KSPACE + 1];
  double cs[OVS_MAX_KSPACE], sn[OVS_MAX_KSPACE];
  double y[OVS_MAX_KSPACE];
  double partials[4 * OVS_RED_BLOCKS];
  double scal[8];     // misc scalar results (norms)
  double sc[OVS_MAX_KSPACE + 1];   // scale of each basis slot (1 / norm of what it holds)
};

// one boundary of setBCs_NSVOF / setBCs_Tem with its types (read by FACE_ID)
// and values (read by boundary number) resolved on the host
struct BcBound {
  int off = 0, n = 0;        // node range in bc_nodes
  int ut[3] = {0, 0, 0};     // BCugType(FACE_ID, d)
  double uv[3] = {0, 0, 0};  // BCugValu(b, d)
  int pt = 0, tt = 0;        // BCphigType(FACE_ID), BCTgType(FACE_ID)
  double pv = 0, tv = 0;     // BCphigValu(b), BCTgValu(b)
};

struct SysStore {
  void* vals = nullptr;   // nnz * nv values (internal slot layout)
  void* rhs = nullptr;    // nf * N, field-major
  void* binv = nullptr;   // preconditioner: N*9 (+N pinv +N lsinv), same precision
  bool have_mat = false, have_rhs = false;
};

struct ovs_ctx {
  int device = 0;
  int num_sms = 148;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  cudaStream_t sol_stream = nullptr;             // uploads of a start vector beside the Krylov cycle (SolFeed)
  cudaEvent_t ev_sol = nullptr;
  cudaEvent_t ev_poll[2] = {nullptr, nullptr};   // the done word of a batch of Krylov iterations has arrived
  int N = 0, E = 0, nshl = 0;
  // mesh
  int* ien = nullptr;        // E*nshl, element-major, 0-based
  int* elm_id = nullptr;     // E
  uint8_t* ibc = nullptr;    // N bit masks (bit d <=> IBC(:,d+1) == 1)
  // pattern
  int* rowptr = nullptr;     // N+1, 0-based
  int* colidx = nullptr;     // nnz
  int* diag = nullptr;       // N: slot of the diagonal entry
  int* n2e_ptr = nullptr;    // N+1
  int* n2e = nullptr;        // nshl*E: (element << 3) | local index, sorted by element
  int* tmap = nullptr;       // nnz: slot of (j, i) for slot (i, j), transposed solves
  void* vals_t = nullptr;    // transposed FP64 values of the temperature system
  double* vjp_cot = nullptr; // residual VJP work: cotangent, element terms, nodal result
  double* vjp_ge = nullptr;
  double* vjp_grad = nullptr;
  int* row_order = nullptr;  // N: rows in Morton order of the node coordinates (the row pass's order)
  int4* row_rec = nullptr;   // N: per row in that order {A, rowptr[A], n2e_ptr[A], deg | sd << 8 | ne << 16}
  int* row_pos = nullptr;    // N: the place of a node's row in that order
  int* ien_t = nullptr;      // ien and elm_id in the storage order of the element summaries
  int* elm_t = nullptr;      //   (pattern.cu: build_elem_order)
  int* n2e_t = nullptr;      // n2e with the place t of the element for its id
  // edges of the tet edge pass (pattern.cu: build_edges)
  int4* edge_rec = nullptr;      // per edge {A, B, slot of (A, B), slot of (B, A)}, tile by tile of rows
  unsigned* edge_ptr = nullptr;  // edges + 1: offsets into edge_list
  unsigned* edge_list = nullptr; // 6 E entries (t << 4) | (la << 2) | lb, ascending element id per edge
  unsigned* tile_edge = nullptr; // first edge of every tile of OVS_TILE_ROWS rows, and the end
  unsigned* n2s = nullptr;   // nshl*E entries: slots of the element's nodes in the row, one byte each
                             // (one word per entry for tets, two for hexahedra)
  int nnz = 0;
  int max_deg = 0, max_elem = 0;
  // boundary faces of the face assemblies (ovs_set_faces)
  int nface = 0, nfnode = 0, face_flags_all = 0;
  int* face_e = nullptr;      // nface owning elements, 0-based
  int* face_info = nullptr;   // nface: (FACE_OR - 1) | flags << 2
  double* face_h = nullptr;   // nface pairs (h, T_inf)
  int* fnode = nullptr;       // nfnode nodes touched by a face element, ascending
  int* fnode_ptr = nullptr;   // nfnode + 1
  int* fnode_ent = nullptr;   // 4 nface entries (face << 2) | local node, ascending face per node
  void* fbuf[2] = {nullptr, nullptr};   // per-face element arrays, per precision
  // streaming time steps (streaming.cu): staged field buffers, copy streams
  double* stage[OVS_F_COUNT] = {};
  unsigned staged_mask = 0;
  double* rhs_out[4] = {};                // FP64 read-back buffer per system
  cudaStream_t up_stream = nullptr, up_stream2 = nullptr, down_stream = nullptr;
  cudaEvent_t ev_staged = nullptr, ev_staged2 = nullptr, ev_commit = nullptr, ev_rhs_ready = nullptr;
  cudaEvent_t ev_rhs_out[4] = {};         // the last read-back of rhs_out[sys] done
  // hex tensor-core pass (FP32 NS+VOF): off unless OVS_HEX_TC=1 or OVS_OPT_HEX_TC
  int hex_tc = 0;
  // FP64 element pass: node records in registers (0) or shared memory (1);
  // -1 (default): shared memory for NS+VOF, registers for the others, the
  // faster of the two measured for each
  int elem_smem = -1;
  // OVS_MIXED: FGMRES(m) outer over FP32 inner cycles (m = mixed_outer > 0,
  // default 30) or the restarted refinement (0)
  int mixed_outer = 30;
  void* fg_buf = nullptr;    // the flexible outer's basis and directions
  size_t fg_bytes = 0;
  void* hex_kbuf = nullptr;              // E x 64 x 24 block values
  float* hex_w = nullptr;                // W hi + lo, canonical layout
  // boundary-condition producers (ovs_set_bc_spec)
  bool have_bcs = false;
  int* bc_nodes = nullptr;               // BNODES of all boundaries, 0-based
  uint8_t* bc_n101 = nullptr;            // NodeID == 101 per node (or null)
  std::vector<BcBound> bc_bounds;        // in NBOUND order
  // nodal state (FP64, reference layout)
  double* field[OVS_F_COUNT] = {};
  // alpha-stage node records (16 values per node), per precision
  void* rec[2] = {nullptr, nullptr};
  // per-element summaries of the element pass, per precision
  void* esum[2] = {nullptr, nullptr};
  // systems [sys][prec]
  SysStore sys[4][2];
  // last solution of each system (FP64, field-major)
  double* sol[4] = {};
  // GMRES / solve workspace
  GmresDev* gm = nullptr;
  void* basis[2] = {nullptr, nullptr};   // Krylov basis per precision
  size_t basis_bytes[2] = {0, 0};
  double* work64 = nullptr;              // 3 vectors of 5N doubles (b, r, x)
  double* wvec = nullptr;                // P^-1 rhs in FP64, before it becomes the first basis vector
  double* coop_part = nullptr;           // partial sums of the cooperative Arnoldi kernels, then T = (I + L)^-1
  size_t coop_bytes = 0;                 //   (rows of kspace, strictly lower part)
  bool arnoldi_fused = false;            // one-launch Arnoldi variant (env OVS_ARNOLDI_FUSED=1)
  // status words: [0] negative DetJ count, [1] non-finite flag, [3] face column missing from a row
  int* flags = nullptr;
  unsigned long long* cfl_bits = nullptr;
  // pinned host mirror
  int* h_pinned = nullptr;
  double* h_pinned_d = nullptr;
  // ovs_assemble_async: status words and CFL bits of the queued passes, read
  // by ovs_assemble_wait (page-locked, OVS_ASYNC_SLOTS entries)
  bool defer_status = false;
  int async_n = 0;
  int* h_async_flags = nullptr;
  unsigned long long* h_async_cfl = nullptr;
  ovs_params params{};
  bool have_mesh = false, have_pattern = false, have_params = false;
  long long launches = 0;                // kernels launched by this context
  double last_ms = 0.0;                  // device time of the last top-level call
};

// ------------------------------------------------------------ helpers
int ovs_ensure(void** p, size_t bytes);
int ovs_activate(ovs_ctx* c);

// pattern.cu
int ovs_pattern_build(ovs_ctx* c);
int ovs_pattern_to_host(ovs_ctx* c, int* col, int* row);
int ovs_slot_map_to_host(ovs_ctx* c, int* lmap);

// assemble.cu
int ovs_assemble_impl(ovs_ctx* c, int kernel, int tensor_flag, int prec,
                      double* cfl);

// assemble.cu: W operand and block buffer of the hex tensor-core pass
int hex_tc_prepare(ovs_ctx* c);

// streaming.cu
void ovs_streaming_free(ovs_ctx* c);

// faces.cu
int ovs_faces_set_impl(ovs_ctx* c, int nface, const int* f2e, const int* face_or, const int* flags,
                       const double* hconv, const double* tinf);
int ovs_faces_assemble(ovs_ctx* c, int kernel, int prec, int mat, int vec);
void ovs_faces_free(ovs_ctx* c);

// bcs.cu
int ovs_apply_bcs_impl(ovs_ctx* c, int which);
void ovs_bcs_free(ovs_ctx* c);

// spmv.cu / gmres.cu
int ovs_precond_setup(ovs_ctx* c, int sys, int prec);
int ovs_spmv_impl(ovs_ctx* c, int sys, int prec, const double* dx,
                  double* dy);
int ovs_spmv_pre_impl(ovs_ctx* c, int sys, int prec, const double* dx, double* dy);
int ovs_spmv_rows_impl(ovs_ctx* c, int sys, int prec, bool precond, const double* dx, double* dy, const int* rows,
                       int nrows);
int ovs_precond_apply_impl(ovs_ctx* c, int sys, int prec, const double* dx, double* dy);
// The start vector of a cycle on its way from the host: columns of N values, in
// any memory, to dst (column-major).  A cycle needs it for the last update only,
// so the host copies it in pieces between the launches of the cycle's steps
// (sol_stream), and touches the pages of `out`, the columns where the result will land.
struct SolFeed {
  const double* const* cols;
  int ncol;
  size_t n;            // values per column
  double* dst;
  double* const* out;  // host columns whose pages to touch (null: none)
  size_t at = 0;       // values sent so far
};
// queue the next `count` values (of n * ncol; every one left for 0)
int ovs_feed(ovs_ctx* c, SolFeed* f, size_t count);
int ovs_gmres_ref_impl(ovs_ctx* c, int sys, double tol, int kspace, int kmin,
                       double* dsol, ovs_gmres_info* info, SolFeed* feed = nullptr);
int ovs_solve_impl(ovs_ctx* c, int sys, int mode, double rtol, int kspace,
                   int max_cycles, ovs_solve_info* info);
int ovs_round_impl(ovs_ctx* c, int sys);
int ovs_update_impl(ovs_ctx* c, int sys);
int ovs_resnorm_impl(ovs_ctx* c, int prec, double r[4]);
int ovs_profile_assemble(ovs_ctx* c, int kernel, int prec, int reps, double* ms, int parts);
int ovs_residual_vjp_impl(ovs_ctx* c, int kernel, const double* cot_host, double* grad_host);
int ovs_gmres_transposed_impl(ovs_ctx* c, int sys, const double* drhs, double tol, int kspace, int kmin,
                              double* dsol, ovs_gmres_info* info);
int ovs_profile_krylov(ovs_ctx* c, int what, int sys, int prec, int reps, double* ms);

// launch geometry helper
static inline int ovs_grid(size_t n, int threads, int cap) {
  size_t g = (n + threads - 1) / threads;
  if (g < 1) g = 1;
  if (g > (size_t)cap) g = cap;
  return (int)g;
}
