// Internal declarations shared by the host code and the CUDA kernels of
// liblbm.so.  Not part of the public ABI (include/lbm.h is).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <vector>

#include "lbm.h"

namespace lbm {

constexpr int kQ = 19;

// ---------------------------------------------------------------- D3Q19 set
// Velocity set and opposite directions of the reference (SP3:167-180).
__host__ __device__ constexpr int cx(int q) {
  return (q == 1 || q == 7 || q == 9 || q == 15 || q == 17) ? 1
         : (q == 2 || q == 8 || q == 10 || q == 16 || q == 18) ? -1
                                                                : 0;
}
__host__ __device__ constexpr int cy(int q) {
  return (q == 3 || q == 7 || q == 8 || q == 11 || q == 13) ? 1
         : (q == 4 || q == 9 || q == 10 || q == 12 || q == 14) ? -1
                                                                 : 0;
}
__host__ __device__ constexpr int cz(int q) {
  return (q == 5 || q == 11 || q == 12 || q == 15 || q == 16) ? 1
         : (q == 6 || q == 13 || q == 14 || q == 17 || q == 18) ? -1
                                                                  : 0;
}
__host__ __device__ constexpr int opp(int q) {
  return q == 0 ? 0 : (q <= 6 ? (q % 2 ? q + 1 : q - 1) : (q <= 10 ? 17 - q : (q <= 14 ? 25 - q : 33 - q)));
}
__host__ __device__ constexpr double weight(int q) {
  return q == 0 ? 1.0 / 3.0 : (q <= 6 ? 1.0 / 18.0 : 1.0 / 36.0);
}

// d'Humieres moment basis of the reference (SP3:64-83) as polynomials of the
// velocity components; row k, column q.
__host__ __device__ constexpr int mcoef(int k, int q) {
  const int x = cx(q), y = cy(q), z = cz(q);
  const int c2 = x * x + y * y + z * z;
  switch (k) {
    case 0: return 1;
    case 1: return 19 * c2 - 30;
    case 2: return (21 * c2 * c2 - 53 * c2 + 24) / 2;
    case 3: return x;
    case 4: return (5 * c2 - 9) * x;
    case 5: return y;
    case 6: return (5 * c2 - 9) * y;
    case 7: return z;
    case 8: return (5 * c2 - 9) * z;
    case 9: return 3 * x * x - c2;
    case 10: return (3 * c2 - 5) * (3 * x * x - c2);
    case 11: return y * y - z * z;
    case 12: return (3 * c2 - 5) * (y * y - z * z);
    case 13: return x * y;
    case 14: return y * z;
    case 15: return x * z;
    case 16: return (y * y - z * z) * x;
    case 17: return (z * z - x * x) * y;
    default: return (x * x - y * y) * z;
  }
}
// Squared norm of row k (rows are mutually orthogonal, so M^-1 = M^T diag(1/norm)).
__host__ __device__ constexpr int mnorm(int k) {
  int s = 0;
  for (int q = 0; q < kQ; q++) s += mcoef(k, q) * mcoef(k, q);
  return s;
}
// Opposite pairs (q, opp q) with q the first of the pair in index order.
__host__ __device__ constexpr int pair_q(int i) {
  return i == 0 ? 1 : i == 1 ? 3 : i == 2 ? 5 : i == 3 ? 7 : i == 4 ? 8 : i == 5 ? 11 : i == 6 ? 12 : i == 7 ? 15 : 16;
}
// even moments: symmetric under e -> -e; odd: antisymmetric.
__host__ __device__ constexpr bool even_moment(int k) {
  return !(k == 3 || k == 4 || k == 5 || k == 6 || k == 7 || k == 8 || k == 16 || k == 17 || k == 18);
}

// ---------------------------------------------------------------- constants
struct MrtConstants {
  double M[kQ][kQ];
  double MI[kQ][kQ];  // Gauss-Jordan inverse, bit-identical to the reference's
  double S[kQ];
  double s_v, s_o;
};
// Rates for a lattice of spacing dx and time step dt (the reference's init:
// lat_c = dx / dt, c_s2 = lat_c^2 / 3, tau = nu / (c_s2 dt) + 0.5); dx = dt = 1
// is the default lattice.
bool build_mrt_constants(double nu, MrtConstants* out, double dx = 1.0, double dt = 1.0);

// Self-defined lattice velocity (lattice_v with dx, dt; SP3:1286-1296,
// 1326-1330, 1382-1394, 1423-1500, 2414-2439): the discrete velocities are
// e lat_c, the equilibrium divides by c2 = lat_c^2 and c4 = c2^2, the Guo
// force by c_s2 and c_s2^2, the forcing enters the moments as dt F and the
// velocity as dt g / 2.  on = 0 is the default lattice (lat_c = dt = 1),
// for which the kernels keep their unit-lattice arithmetic.
struct Lattice {
  int on = 0;
  double c = 1.0;              // lat_c = dx / dt
  double ic = 1.0;             // 1 / lat_c
  double cs2 = 1.0 * 1.0 / 3;  // c_s^2 = lat_c^2 / 3
  double c2 = 1.0, c4 = 1.0;   // lat_c^2, lat_c^4 (feq)
  double dt = 1.0, dx = 1.0;
};
Lattice make_lattice(double dx, double dt);

// ---------------------------------------------------------------- geometry
struct Geometry {
  int nx = 0, ny = 0, nz = 0;
  int count = 0;                 // fluid nodes
  int npad = 0;                  // SoA stride (multiple of 256)
  double porosity = 0.0;         // over the permeability window
  std::vector<int32_t> coor;     // [count+1], ref id -> i*ny*nz + j*nz + k
  std::vector<int32_t> ref_of;   // [count], internal index -> ref id (1-based)
  std::vector<int32_t> int_of;   // [count+1], ref id -> internal index (row 0 = -1)
  std::vector<int32_t> src;      // [18][npad], pull sources (flat index q*npad + m)
  std::vector<uint8_t> in_window;// [count] internal order; empty = whole box
  int window_volume = 0;
};

// Fluid-node compaction in the reference order (SP3:1018-1071).
void compact_reference(const uint8_t* mask, int nx, int ny, int nz, Geometry* g);
// Internal ordering: fills ref_of / int_of for the requested curve.
void order_nodes(const uint8_t* mask, int ordering, Geometry* g);
// Pull table in internal order with halfway bounce-back resolved.
void build_pull_table(const uint8_t* mask, Geometry* g);
// Push table nei_loc (reference form) from the pull table.
void pull_to_push(const Geometry& g, int32_t* nei_loc);
void set_window(const int window[6], Geometry* g);

// ------------------------------------------------- pressure/velocity faces
// One boundary operation on the post-streaming populations F of a face node,
// in the reference's program order (boundary_pressure then
// boundary_velocity).  nb / nb4 are snapshot slots (internal index -
// snap_begin) of the nodes whose previous-step state the rule reads, -1 for
// none (the reference's row 0, zero).
enum BcKind : int8_t {
  kBcPressureRest = 0,    // F = f_eq(rho_b, 0)
  kBcPressureNbU = 1,     // F = f_eq(rho_b, u[nb])
  kBcPressureMoment = 2,  // F = MI (M f[nb] with m_0 = rho_b)
  kBcPressureNeq = 3,     // F = f_eq(rho_b, u[nb]) + f[nb4] - f_eq(rho[nb], u[nb])
  kBcVelocityEq = 4,      // F = f_eq(1, u_b)
  kBcVelocityNeq = 5,     // incoming q: F_q = f_eq(opp q; 1, u_b) - F_opp q + f_eq(q; 1, u_b)
  kBcVelocityNbRho = 6,   // F = f_eq(rho[nb], u_b)
};
struct BcOp {
  int8_t kind;
  int8_t face;  // INPUT.dat face index 0..5 = xp, xn, yp, yn, zp, zn (density / velocity of the rule)
  int8_t axis;  // kBcVelocityNeq: axis of the incoming test
  int8_t sign;  // kBcVelocityNeq: +1 -> q with e_axis < 0 are incoming, -1 -> e_axis > 0
  int32_t nb;
  int32_t nb4;
};
// Node classes after bc_partition, in internal order:
//   [0, snap_begin)          interior nodes (no boundary involvement)
//   [snap_begin, n_main)     nodes whose state a boundary rule reads
//   [n_main, count)          nodes a boundary rule writes (face nodes)
// The main step kernel runs over [0, n_main) and records the post-streaming
// state of [snap_begin, n_main); the boundary kernel runs over [n_main, count).
struct BcPlan {
  bool active = false;
  int n_main = 0, snap_begin = 0;
  std::vector<int32_t> op_off;  // [count - n_main + 1] CSR over boundary nodes
  std::vector<BcOp> ops;
};
bool bc_active(const lbm_boundary& bc);
// Reorders g (ref_of / int_of) into the three classes, keeping the order
// within each class, and builds the per-node operation lists.
void bc_partition(const uint8_t* mask, const lbm_boundary& bc, Geometry* g, BcPlan* plan);
// The same program without reordering: the written nodes (internal indices)
// with their operations (CSR, program order per node) and the nodes whose
// state the operations read; BcOp.nb / nb4 index snap_nodes (-1 = none).
struct BcLists {
  std::vector<int32_t> nodes, op_off, snap_nodes;
  std::vector<BcOp> ops;
};
void bc_node_lists(const lbm_boundary& bc, const Geometry& g, BcLists* out);

// Two pinned staging buffers for device -> pageable host copies; copies
// borrow them from a process-wide pool per device (transfer.cpp).
struct PinnedStage {
  static constexpr size_t kChunk = size_t(16) << 20;
  void* buf[2] = {nullptr, nullptr};
  cudaEvent_t ev[2] = {nullptr, nullptr};
  PinnedStage() = default;
  PinnedStage(const PinnedStage&) = delete;
  PinnedStage& operator=(const PinnedStage&) = delete;
  ~PinnedStage();
};
// Copies `bytes` from device memory `src` to host memory `dst` in order on
// `st` (a stream of the current device) and returns when the host copy is
// complete.
struct HostPart {
  void* dst;
  size_t bytes;
};
// (several destinations: their sources follow one another at src)
cudaError_t d2h_staged(const HostPart* parts, int nparts, const void* src, cudaStream_t st);
inline cudaError_t d2h_staged(void* dst, const void* src, size_t bytes, cudaStream_t st) {
  const HostPart one{dst, bytes};
  return d2h_staged(&one, 1, src, st);
}
// Pins one stage for the current device if its pool has none yet (so that
// the process's first field read does not pay for it).  Where no memory can be
// pinned the reads go without.
void stage_pool_prime();

// Device memory of the solvers, from the current device's default memory
// pool with its release threshold raised: what a destroyed solver frees
// stays mapped in the process, and the next solver of a similar size takes
// it without new mappings.  dev_free first waits for the device to go idle,
// as cudaFree does, so that no launch in flight can still use the memory.
cudaError_t dev_alloc(void** p, size_t bytes);
void dev_free(void* p);
// Returns the memory freed solvers left in the pools to the driver.
cudaError_t dev_pool_trim();

// A device buffer of a solver.  After an allocation that failed it is empty
// (p null, bytes 0), so a caller that decides by either allocates again.
struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() { release(); }
  void release() {
    if (p) dev_free(p);
    p = nullptr;
    bytes = 0;
  }
  cudaError_t alloc(size_t b) {
    release();
    if (b == 0) return cudaSuccess;
    const cudaError_t e = dev_alloc(&p, b);
    if (e == cudaSuccess)
      bytes = b;
    else
      p = nullptr;
    return e;
  }
  template <typename T>
  T* as() const {
    return static_cast<T*>(p);
  }
};

// Mask and box of a single-phase handle (for solvers coupled to it).
const uint8_t* lbm_internal_mask(lbm_handle* h, int* nx, int* ny, int* nz);
extern "C" const uint8_t* lbm_cg_internal_mask(lbm_cg_handle* h, int* nx, int* ny, int* nz);

// ---------------------------------------------------------------- errors
void set_error(const std::string& msg);
lbm_status fail(lbm_status s, const std::string& msg);

#define LBM_CUDA_TRY(expr)                                                               \
  do {                                                                                   \
    cudaError_t _e = (expr);                                                             \
    if (_e != cudaSuccess)                                                               \
      return ::lbm::fail(_e == cudaErrorMemoryAllocation ? LBM_ERR_OOM : LBM_ERR_CUDA,   \
                         std::string(#expr) + ": " + cudaGetErrorString(_e));            \
  } while (0)

// ---------------------------------------------------------------- kernels
// Storage kinds of the population arrays.
enum class Store { F64 = 0, F32 = 1, F16 = 2, F64D = 3 };

// Phase of an in-place population array (kernels_common.cuh): where the
// post-streaming f_q(p) of the state lies, and where a step leaves the next
// state's.
enum Phase { kPull = 0, kLocal = 1 };

struct StepArgs {
  void* pop;             // [19][npad] populations, updated in place
  int phase;             // Phase of the state the step starts from
  const int32_t* table;  // [18][npad]
  const int32_t* rows;   // FP32: [9][npad] row form of the table (row_table.cuh), or null
  int ahead;             // nodes ahead that a block prefetches into L2, 0 = none
  int chained;           // launched as a programmatic dependent of the step before it
  int carveout;          // percent of an SM's L1 to ask for as shared memory, 0 = the driver's choice
  int n;                 // fluid nodes
  int npad;
  // macro input for a step that must use given rho/u (first step after init
  // or restart); null otherwise
  const void* rho_in;
  const void* u_in;      // [3][npad]
  // macro output of this step's pre-collision rho/u; null = not written
  void* rho_out;
  void* u_out;           // [3][npad]
  double gx, gy, gz;
  double s_v, s_o;
  double fp16_scale;
  float fp16_inv;        // (float)(1 / fp16_scale): a division in double per thread else
  // pressure/velocity faces: nodes [n_main, n) are left to the boundary
  // kernel; nodes [snap_begin, n_main) record their post-streaming state in
  // snap_dst ([23][nsnap] doubles: f_0..f_18, rho, ux, uy, uz; slot = p -
  // snap_begin).  Without faces n_main = n and snap_dst = null.
  int n_main;
  int snap_begin;
  int nsnap;
  double* snap_dst;
  // compact pull table (null = read `table`): per aligned warp of 32 nodes
  // and direction q a base node index ct_base[(q-1)*nwarps + w] (-1: the
  // warp reads `table` for q) and per node a 16-bit offset from it (0xFFFF:
  // halfway bounce-back, source opp(q)*npad + p); offsets of directions
  // 2i+1, 2i+2 share one 32-bit word, ct_off as [9][npad][2]
  const int32_t* ct_base;
  const uint16_t* ct_off;
  int nwarps;
  // lattice of the step.  The FP64 reference kernel takes g above as given
  // and does the reference's lattice arithmetic; the deviation-storage
  // kernels work in units of lat_c (g above is dt g / lat_c, the macro
  // arrays rho_in/u_in/u_out hold the velocity itself: read times 1/lat_c,
  // written times lat_c)
  Lattice lat;
};
// Nodes per block of the step where the caller asked for no size: 64 for small
// solves, whose few large blocks leave SMs idle or give some twice the work of
// others, and for the bit-exact FP64 step, whose blocks keep the FP64 pipe
// busier when they end one by one.  (One thread per node; half as many threads
// where a thread takes two nodes.)  us per step, 64 | 256 threads:
// FP64 5 K nodes 4.28 | 5.66, 92 K 11.5 | 12.3, 310 K 28.2 | 30.9, 5.9 M 504 | 529;
// FP64 deviation 5 K 2.15 | 3.00, 310 K 13.3 | 14.3, 734 K 45.5 | 43.8; FP32 5 K
// 1.85 | 2.32, 49 K 3.12 | 3.51, 131 K 4.79 | 5.30 (above that two nodes per
// thread, 310 K 7.99 | 7.82).
//
// Beside a face kernel (faces) the FP64 step's smaller blocks would spread over
// the face kernel's SMs as well: 256 | 128 | 64, FP64 with pressure faces, 70 K
// nodes 19.0 | 19.2 | 20.4, 105 K 20.7 | 21.7 | 22.3, 149 K 25.4 | 24.4 | 24.6,
// 354 K 49.9 | 46.6 | 48.4; FP32 (256 | 128 | 64) 34 K 4.0 | 3.9 | 3.85, 105 K
// 5.7 | 5.6 | 5.9, 149 K 6.8 | 6.7 | 6.9.
constexpr int default_block(Store kind, long long n, bool faces = false) {
  if (faces && kind == Store::F64) return n < 148 * 850 ? 256 : 128;
  if (faces && (kind == Store::F32 || kind == Store::F16) && n >= 148 * 512 && n < 148 * 1024) return 128;
  return kind == Store::F64 || n < (kind == Store::F64D ? 400000 : 148 * 1024) ? 64 : 256;
}

cudaError_t launch_step(Store kind, const StepArgs& a, int block, cudaStream_t st);
// Builds the compact pull table from `table` ([18][npad], n fluid nodes);
// counts the (warp, direction) pairs left on the full table in *wide (device).
cudaError_t launch_compact_table(const int32_t* table, int n, int npad, int32_t* ct_base, uint16_t* ct_off,
                                 unsigned long long* wide, cudaStream_t st);

// Row form of a table of row stride `stride`, its first n nodes; adds the
// marked nodes to *marked (device).
cudaError_t launch_row_table(const int32_t* table, int stride, int n, int32_t* rows, int* marked, cudaStream_t st);
// Where the row form is the better one to read: in the FP32 single-phase step
// and the D3Q19 solutes, for n nodes with pop_bytes of populations per node
// (rows_large: whether to build it), `marked` of them marked (rows_pay: whether
// to keep and read it).
//  * It reads 36 bytes per node against 72, for arithmetic that the other
//    steps have no room for.  us per step, rows | int32, 256^3, porosity 0.35:
//    FP32 166 | 173, FP16 129 | 125 (0.6: 226 | 216), FP64 717 | 671, FP64
//    deviation 323 | 317 (0.6: 562 | 544); D3Q19 solute 192^3 FP32 111 | 113,
//    FP64 211 | 220; pools of 96^3 to 200^3 1 to 8 % slower with rows.
//  * A warp with a marked node waits for up to five table entries more, and
//    about every warp has one where a row of cells holds fewer than 32 nodes.
//    Reference order marks 2 / nx of the nodes, the curve orders most of them.
//    FP32 us, rows | int32, nx = 64, 96, 128, 256: porosity 0.35 (1.1 M nodes) 34.8 |
//    34.5, 33.6 | 34.4, 32.7 | 34.8, 31.0 | 34.3; 0.6 (1.9 M) 63.9 | 59.6, 60.0 | 59.9,
//    60.2 | 61.4, 58.1 | 59.3: the line is drawn at nx = 100.
//  * Its arithmetic costs more than the bytes it saves while the solve lives
//    in the 126 MB L2 with either form: FP32 cubes at porosity 0.35 took (int32
//    | rows) 9.12 | 9.51 us at 96^3, 12.8 | 13.4 at 112^3 (73 MB with the int32
//    table), 21.1 | 19.4 at 128^3 (109 MB).
constexpr bool rows_large(long long n, long long pop_bytes) { return n * (pop_bytes + 72) > (90LL << 20); }
constexpr bool rows_pay(long long marked, long long n) { return marked * 50 <= n; }
// Nodes ahead of its own that a block prefetches into L2, or 0 for a solve that
// stays in L2, for pop_bytes of rows and table_bytes of table per node.  A step
// waits on two loads in a row, table then populations; asked for early, both
// come from L2.  What matters is how much is on its way: too little and the
// lines arrive late, too much and they are evicted again.  The best distance
// was about 44 KB per SM for every step (a multiple of 64 nodes per SM).  us per
// step without | at that | at 640 nodes per SM, cubes at porosity 0.35: FP32 256^3
// (112 bytes) 174 | 161 | 161, FP16 256^3 (110) 136 | 128 | 128, FP64 deviation 256^3
// (224) 335 | 299 | 314, D3Q7 FP32 192^3 (60) 33.1 | 27.6 | 27.6, FP64 192^3 (96) 60.4
// | 48.0 | 48.0, D3Q19 FP32 192^3 (124) 94.4 | 77.6 | 78.3, FP64 128^3 (212) 53.2 | 44.7
// | 48.5.  The bit-exact FP64 step is bound by its FP64 pipe: 484 to 491 at any.
constexpr int prefetch_ahead(long long n, long long pop_bytes, long long table_bytes) {
  const long long bytes = pop_bytes + table_bytes;
  return n * bytes > (120LL << 20) ? 148 * 64 * (int)((44000 / bytes + 32) / 64) : 0;
}

// Whether successive steps are launched as programmatic dependents
// (kernels_common.cuh), for n nodes.  The next step's blocks then start in the
// slots the running one leaves, which saves a launch gap per step, but where
// the two together neither leave SMs free nor fill them they land unevenly.  us
// per step at the default block size, chained | not, porosity 0.35:
//   FP32  10 K nodes 1.93 | 2.38, 21 K 2.19 | 2.63, 37 K 2.63 | 3.00, 49 K 3.30 | 3.26,
//         71 K 4.03 | 3.66, 102 K 4.99 | 4.43, 126 K 5.25 | 4.96, 157 K 5.39 | 5.58, 310 K
//         7.78 | 8.09, 734 K 17.3 | 18.1 (FP16 the same within 6 %)
//   FP64  10 K 5.30 | 5.84, 18 K 5.91 | 6.23, 22 K 6.90 | 6.13, 32 K 7.87 | 6.48, 53 K
//         8.79 | 7.62, 66 K 8.95 | 8.78, 71 K 8.46 | 9.15, 126 K 13.2 | 13.8, 734 K
//         65.8 | 67.6
// FP64 deviation storage gains 2 to 20 % and loses up to 3 % about 20 K; the
// solutes (st7_api.cpp) gain at every size.  Larger blocks that were asked for
// gain nearly everywhere (256 nodes, FP64 39 K 8.40 | 8.65, FP32 92 K 3.92 | 4.31).
constexpr bool chain_pays(Store kind, long long n, int block) {
  return kind == Store::F64D || block >= 256 ||
         (kind == Store::F64 ? n <= 148 * 128 || n >= 148 * 480 : n <= 148 * 256 || n >= 148 * 1024);
}

constexpr int kSnapRows = kQ + 4;  // per-step record of a node: f_0..f_18, rho, ux, uy, uz

// Boundary kernel: the face nodes [n_main, n) of one step (pull, rules, macro,
// record, collide) or, with bnd_f set, only the post-rule populations of the
// current state ([19][n - n_main] doubles) for reductions and exports.
struct BcArgs {
  StepArgs s;               // pops, table, macro in/out, rates, n_main, snap_begin, nsnap, snap_dst
  const double* snap_src;   // the previous step's record
  const int32_t* op_off;
  const BcOp* ops;
  const double* mi;         // [19*19] M^-1 (kBcPressureMoment)
  double face_rho[6];
  double face_u[6][3];
  double* bnd_f;            // finalize mode output, or null
};
cudaError_t launch_boundary(Store kind, const BcArgs& a, cudaStream_t st);

struct ReduceArgs {
  const void* pop;        // [19][npad] populations of the state
  int phase;              // its Phase
  const int32_t* table;
  int n, npad;
  const void* rho_in;     // when the state is "given" (no step since set): use these
  const void* u_in;
  const void* u_prev;     // [3][npad] velocity one step earlier (null -> zero change)
  int last_p;             // internal index of the reference's last node (excluded from Error)
  const uint8_t* window;  // [n] or null
  double gx, gy, gz;
  double fp16_scale;
  double* rho_out;        // optional double[n] (internal order)
  double* u_out;          // optional double[3][npad]
  double* partials;       // [blocks][8]
  double* result;         // [8]
  int n_main;             // nodes [n_main, n) read their populations from bnd_f
  const double* bnd_f;    // [19][n - n_main] post-rule populations, or null
  Lattice lat;            // as StepArgs::lat (gx.. follow the same convention)
};
// result: t1, t2, t3, umax2, Qx, Qy, Qz, mass
cudaError_t launch_reduce(Store kind, const ReduceArgs& a, cudaStream_t st);
int reduce_blocks(int n);

// f[(count+1)*19] reference AoS <-> device storage
cudaError_t launch_export_pop(Store kind, const void* pop, int phase, const int32_t* table, const int32_t* ref_of,
                              int n, int npad, double fp16_scale, double* out, cudaStream_t st,
                              int n_main = 0, const double* bnd_f = nullptr);
// (the imported state is a kPull state)
cudaError_t launch_import_pop(Store kind, void* pop, const int32_t* table, const int32_t* ref_of, int n,
                              int npad, double fp16_scale, const double* in, cudaStream_t st);
// rho/u reference-layout doubles -> device macro arrays of the storage's type
cudaError_t launch_import_macro(Store kind, void* rho, void* u, const int32_t* ref_of, int n, int npad,
                                const double* rho_in, const double* u_in, cudaStream_t st);
cudaError_t launch_export_macro(const double* rho_int, const double* u_int, const int32_t* ref_of, int n,
                                int npad, double* rho_ref, double* u_ref, cudaStream_t st);
// out[0] = 0, out[ref_of[p]] = src[p] as double (FP64 or FP32 source)
cudaError_t launch_export_scalar(bool f64, const void* src, const int32_t* ref_of, int n, double* out, cudaStream_t st);
cudaError_t set_mi_constant(const double* mi361, cudaStream_t st);
// True when M^-1 has the zero / power-of-two pattern the bit-exact FP64
// kernel was compiled for (mi_pattern.h, generated from mrt.cpp).
bool mi_pattern_matches(const double* mi361);
// uniform post-streaming state f_q = feq[q] at every node, a kPull state
// written through the inverse pull so the next step pulls exactly feq
cudaError_t launch_init_uniform(Store kind, void* pop, const int32_t* table, int n, int npad, double fp16_scale,
                                const double* feq19, cudaStream_t st);
cudaError_t launch_fill_macro(Store kind, void* rho, void* u, int n, int npad, double rho0, const double* u3,
                              cudaStream_t st);

size_t store_bytes(Store kind);

}  // namespace lbm
