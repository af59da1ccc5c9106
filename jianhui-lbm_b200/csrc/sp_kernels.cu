// Single-phase fused collide + pull-stream kernels in deviation storage
// (FP32, FP16, FP64-fast) and the dispatch of every single-phase kernel.
//
// One thread owns one fluid node and updates its 19 slots in place
// (kernels_common.cuh).  Per node a step moves, from/to HBM, 19 populations
// in and 19 out (2*19*s bytes, s = bytes per stored population); a step from
// a kPull state gathers and scatters them through 18 int32 table entries
// (72 bytes more), the step after it works on the node's own slots.
#include "bc_kernels.cuh"
#include "collide_vec.cuh"
#include "row_table.cuh"

namespace lbm {

cudaError_t launch_step_f64(const StepArgs& a, int block, cudaStream_t st);
cudaError_t reduce_f64(const ReduceArgs& a, cudaStream_t st);
cudaError_t export_f64(const void*, int, const int32_t*, const int32_t*, int, int, double*, cudaStream_t, int,
                       const double*);
cudaError_t launch_boundary_f64(const BcArgs& a, cudaStream_t st);
cudaError_t import_f64(void*, const int32_t*, const int32_t*, int, int, const double*, cudaStream_t);
cudaError_t import_macro_f64(void*, void*, const int32_t*, int, int, const double*, const double*, cudaStream_t);

// Compact pull table: per aligned warp of 32 nodes and direction q one int32
// base node index (-1: the warp reads the int32 table for q) and per node a
// 16-bit offset from it (0xFFFF: halfway bounce-back, source opp(q)*npad +
// p), the offsets of directions 2i+1 and 2i+2 packed in one 32-bit word
// ([9][npad] words): 18*2 + 18*4/32 bytes of table per node instead of 72.
__device__ __forceinline__ size_t ct_off_index(int q, int p, int npad) {
  return (size_t)((q - 1) >> 1) * 2 * npad + 2 * (size_t)p + ((q - 1) & 1);
}

// One thread per (node, direction) row of 32 nodes: the warp's fluid sources
// in row q as a base plus 16-bit offsets, or -1 when they spread wider.
__global__ void __launch_bounds__(256) compact_table_kernel(const int32_t* __restrict__ table, int n, int npad,
                                                           int32_t* __restrict__ ct_base,
                                                           uint16_t* __restrict__ ct_off,
                                                           unsigned long long* __restrict__ wide) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;  // npad is a multiple of 256: whole warps
  const int q = blockIdx.y + 1;
  if (p >= npad) return;
  const int32_t e = table[(size_t)(q - 1) * npad + p];
  const bool live = p < n;
  const unsigned m = (unsigned)(e - q * npad);
  const bool fluid = live && m < (unsigned)npad;
  const bool bounce = live && e == opp(q) * npad + p;
  const unsigned lo = __reduce_min_sync(0xffffffffu, fluid ? m : 0xffffffffu);
  const unsigned hi = __reduce_max_sync(0xffffffffu, fluid ? m : 0u);
  const bool odd = __any_sync(0xffffffffu, live && !fluid && !bounce);
  const bool any = lo != 0xffffffffu;
  const bool too_wide = odd || (any && hi - lo > 0xFFFEu);
  const size_t w = p >> 5;
  if ((threadIdx.x & 31) == 0) {
    ct_base[(size_t)(q - 1) * (npad >> 5) + w] = too_wide ? -1 : (any ? (int32_t)lo : 0);
    if (too_wide) atomicAdd(wide, 1ull);
  }
  ct_off[ct_off_index(q, p, npad)] = (too_wide || !fluid) ? (uint16_t)0xFFFF : (uint16_t)(m - lo);
}

cudaError_t launch_compact_table(const int32_t* table, int n, int npad, int32_t* ct_base, uint16_t* ct_off,
                                 unsigned long long* wide, cudaStream_t st) {
  if (npad % 256 != 0) return cudaErrorInvalidValue;
  cudaError_t e = cudaMemsetAsync(wide, 0, sizeof(unsigned long long), st);
  if (e != cudaSuccess) return e;
  compact_table_kernel<<<dim3(npad / 256, 18), 256, 0, st>>>(table, n, npad, ct_base, ct_off, wide);
  return cudaGetLastError();
}

// Whether a thread of an FP32-arithmetic step takes two nodes: from one node
// per thread of a full wave's threads on.  One | two nodes, us per FP32 step:
// 4.28 | 4.35 at 92 K nodes, 5.93 | 5.52 at 179 K, 9.12 | 8.23 at 310 K,
// 21.1 | 18.1 at 734 K, 169 | 164 at 5.9 M; FP16 19.1 | 16.9 and 159 | 137 at
// the last two.
static bool two_nodes(int n) { return n >= 148 * 1024; }

// Where a step reads and writes: the node's own slots (a kLocal state), or
// the slots of the int32 table, of its row form (FP32) or of its compact form
// (a kPull state).  LocalOdd: the node's own slots, of an odd number of nodes
// that face nodes follow: the last pair's second slot is the face kernel's,
// which runs beside the step (asking everywhere costs 0.5 to 3 % in L2).
enum class Slots { Local, LocalOdd, Table, Rows, Compact };

// The block's warp bases of the compact table, in shared memory, and this
// node's offset words: the words are loaded before the barrier so that their
// latency overlaps the bases'.
template <int BS>
struct CompactBlock {
  int32_t base[18][BS / 32];
};
template <int BS>
__device__ __forceinline__ void compact_load(CompactBlock<BS>& cb, const StepArgs& a, int p, uint32_t (&ow)[9]) {
  if (p < a.n_main) {
    const uint32_t* __restrict__ off = reinterpret_cast<const uint32_t*>(a.ct_off);
#pragma unroll
    for (int i = 0; i < 9; i++) ow[i] = __ldg(off + (size_t)i * a.npad + p);
  }
  for (int k = threadIdx.x; k < 18 * (BS / 32); k += BS) {
    const int qq = k / (BS / 32), w = k % (BS / 32);
    const int gw = blockIdx.x * (BS / 32) + w;
    cb.base[qq][w] = gw < a.nwarps ? __ldg(a.ct_base + (size_t)qq * a.nwarps + gw) : -1;
  }
  __syncthreads();
}
template <int BS>
__device__ __forceinline__ void compact_slots(const CompactBlock<BS>& cb, const StepArgs& a, int p,
                                              const uint32_t (&ow)[9], int32_t (&slot)[kQ]) {
  const int wl = threadIdx.x >> 5;
#pragma unroll
  for (int q = 1; q < kQ; q++) {
    const int32_t b = cb.base[q - 1][wl];
    const int o = ((q - 1) & 1) ? (int)(ow[(q - 1) >> 1] >> 16) : (int)(ow[(q - 1) >> 1] & 0xFFFFu);
    int32_t t = 0;
    if (b < 0) t = __ldg(a.table + (size_t)(q - 1) * a.npad + p);
    const int32_t c = o == 0xFFFF ? opp(q) * a.npad + p : q * a.npad + b + o;
    slot[q] = b < 0 ? t : c;
  }
}
// slot[q] of node p through the int32 table or its compact form
template <Slots SL, int BS>
__device__ __forceinline__ void read_slots(const CompactBlock<BS>& cb, const StepArgs& a, int p,
                                           const uint32_t (&ow)[9], int32_t (&slot)[kQ]) {
  if constexpr (SL == Slots::Compact) {
    compact_slots(cb, a, p, ow, slot);
  } else {
#pragma unroll
    for (int q = 1; q < kQ; q++) slot[q] = __ldg(a.table + (size_t)(q - 1) * a.npad + p);
  }
}

// The step in FP64 deviation storage; 16-warp blocks per SM asked of the
// register allocator at 256 threads (128 registers).
template <int BS, bool GIVEN, bool WRITE, Slots SL>
__global__ void __launch_bounds__(BS, BS == 256 ? 2 : 1) step_dev_kernel(StepArgs a) {
  constexpr Store K = Store::F64D;
  const int p = blockIdx.x * BS + threadIdx.x;
  __shared__ SlotKeep<SL == Slots::Local ? 1 : BS, 1> keep;
  __shared__ CompactBlock<SL == Slots::Compact ? BS : 32> cb;
  uint32_t ow[9] = {};
  if constexpr (SL == Slots::Compact) compact_load(cb, a, p, ow);
  prefetch_block<BS, BS, SL == Slots::Table ? 18 : 0>(static_cast<const double*>(a.pop), a.table, a.npad, a.ahead);
  step_begin();
  if (p >= a.n_main) return;
  double* pop = static_cast<double*>(a.pop);
  double f[kQ];
  if constexpr (SL == Slots::Local) {
    step_wait();
#pragma unroll
    for (int q = 1; q < kQ; q++) f[q] = pop[(size_t)opp(q) * a.npad + p];
  } else {
    int32_t slot[kQ];
    read_slots<SL>(cb, a, p, ow, slot);
    step_wait();
#pragma unroll
    for (int q = 1; q < kQ; q++) f[q] = pop[slot[q]];
    keep_slots(keep, threadIdx.x, [&](int q) { return slot[q]; });
  }
  f[0] = pop[p];
  PairSplit<double> ps;
  split_pairs(f, ps);
  double drho, rho, ux, uy, uz;
  // velocities in units of lat_c (1 on the default lattice, where the
  // scalings below are exact)
  if (GIVEN) {
    const double* r = static_cast<const double*>(a.rho_in);
    const double* u = static_cast<const double*>(a.u_in);
    rho = r[p];
    drho = rho - 1.0;
    ux = u[p] * a.lat.ic;
    uy = u[a.npad + p] * a.lat.ic;
    uz = u[2 * a.npad + p] * a.lat.ic;
  } else {
    macro_dev<double>(f, ps, 0.5 * a.gx, 0.5 * a.gy, 0.5 * a.gz, drho, rho, ux, uy, uz);
  }
  if (WRITE) {
    static_cast<double*>(a.rho_out)[p] = rho;
    double* u = static_cast<double*>(a.u_out);
    u[p] = ux * a.lat.c;
    u[a.npad + p] = uy * a.lat.c;
    u[2 * a.npad + p] = uz * a.lat.c;
  }
  if (a.snap_dst != nullptr && p >= a.snap_begin) {
    double full[kQ];
#pragma unroll
    for (int q = 0; q < kQ; q++) full[q] = to_full<K>(f[q], q);
    snap_write(a.snap_dst, a.nsnap, p - a.snap_begin, full, rho, ux, uy, uz);
  }
  mrt_collide_dev<double>(f, ps, drho, rho, ux, uy, uz, a.gx, a.gy, a.gz, a.s_v, a.s_o);
  pop[p] = f[0];
  if constexpr (SL == Slots::Local) {
#pragma unroll
    for (int q = 1; q < kQ; q++) pop[(size_t)q * a.npad + p] = f[q];
  } else {
    for_kept_slots(keep, threadIdx.x, [&](int q, int32_t slot) { pop[slot] = f[opp(q)]; });
  }
}

// Resident blocks per SM asked of the register allocator: one node per
// thread fits 1280 threads (48 registers; given states and the compact table
// spill 4 to 88 bytes), two nodes 640 (96 registers; 512
// threads and 128 registers: 19.6 against 18.4 us at 128^3; 768 threads spill
// 150-230 bytes: 22.9 us).
template <typename V>
constexpr int vec_min_blocks(int bs) {
  return (VecOf<V>::kNodes == 2 ? 640 : 1280) / bs;
}

// The step in FP32 arithmetic (FP32 and FP16 storage): one node per thread
// (V = float) or two (V = F2, collide_vec.cuh).  On its own slots a thread
// takes nodes p and p + 1, which one access loads and stores; through the
// table it takes p and p + 32, so that the lanes of a gather or scatter stay
// on consecutive nodes (with p and p + 1 every one of them would touch twice
// the sectors, half filled).
template <Store K, int BS, typename V, bool GIVEN, bool WRITE, Slots SL>
__global__ void __launch_bounds__(BS, vec_min_blocks<V>(BS)) step_vec_kernel(StepArgs a) {
  using T = typename Traits<K>::T;
  constexpr int N = VecOf<V>::kNodes;
  static_assert(N == 1 || (!GIVEN && SL != Slots::Compact), "given states and the compact table: one node per thread");
  static_assert(N == 2 || SL != Slots::Rows, "the row form: two nodes per thread");
  constexpr bool LOCAL = SL == Slots::Local || SL == Slots::LocalOdd, PAIR = N == 2 && LOCAL;  // p, p + 1
  const int p = N == 1 ? blockIdx.x * BS + threadIdx.x
                : PAIR ? (blockIdx.x * BS + threadIdx.x) * 2
                       : blockIdx.x * BS * 2 + (threadIdx.x >> 5) * 64 + (threadIdx.x & 31);
  const int second = p + (PAIR ? 1 : 32);
  __shared__ SlotKeep<LOCAL ? 1 : BS, N> keep;
  __shared__ CompactBlock<SL == Slots::Compact ? BS : 32> cb;
  uint32_t ow[9] = {};
  if constexpr (SL == Slots::Compact) compact_load(cb, a, p, ow);
  prefetch_block<BS, BS * N, SL == Slots::Rows ? 9 : SL == Slots::Table ? 18 : 0>(
      static_cast<const T*>(a.pop), SL == Slots::Rows ? a.rows : a.table, a.npad, a.ahead);
  step_begin();
  if (p >= a.n_main) return;
  const bool both = N == 2 && second < a.n_main;
  const int p1 = both ? second : p;  // a missing second node is worked on as the first and not stored
  const bool load_both = SL != Slots::LocalOdd || both;
  T* pop = static_cast<T*>(a.pop);
  const float scale = (float)a.fp16_scale;
  const float inv_scale = a.fp16_inv;
  V f[kQ];
  if constexpr (LOCAL) {
    step_wait();
#pragma unroll
    for (int q = 1; q < kQ; q++) load_row<K>(pop + (size_t)opp(q) * a.npad + p, inv_scale, load_both, f[q]);
  } else if constexpr (N == 1) {
    int32_t slot[kQ];  // slot[q] holds f_q on entry and takes f*_opp(q)
    read_slots<SL>(cb, a, p, ow, slot);
    step_wait();
#pragma unroll
    for (int q = 1; q < kQ; q++) f[q] = load_pop_rw<K>(pop + slot[q], inv_scale);
    keep_slots(keep, threadIdx.x, [&](int q) { return slot[q]; });
  } else {
    int32_t s0[kQ], s1[kQ];
    if constexpr (SL == Slots::Rows) {
      int32_t w0[9], w1[9];
#pragma unroll
      for (int i = 0; i < 9; i++) {
        w0[i] = __ldg(a.rows + (size_t)i * a.npad + p);
        w1[i] = __ldg(a.rows + (size_t)i * a.npad + p1);
      }
      row_slots(w0, a.table, a.npad, p, s0);
      row_slots(w1, a.table, a.npad, p1, s1);
    } else {
#pragma unroll
      for (int q = 1; q < kQ; q++) {
        s0[q] = __ldg(a.table + (size_t)(q - 1) * a.npad + p);
        s1[q] = __ldg(a.table + (size_t)(q - 1) * a.npad + p1);
      }
    }
    step_wait();
#pragma unroll
    for (int q = 1; q < kQ; q++)
      f[q] = make_f2(load_pop_rw<K>(pop + s0[q], inv_scale), load_pop_rw<K>(pop + s1[q], inv_scale));
#pragma unroll
    for (int i = 0; i < 9; i++)
      keep.a[i][threadIdx.x] = make_int4(s0[2 * i + 1], s1[2 * i + 1], s0[2 * i + 2], s1[2 * i + 2]);
  }

  if constexpr (N == 1 || PAIR)
    load_row<K>(pop + p, inv_scale, load_both, f[0]);
  else
    f[0] = make_f2(load_pop_rw<K>(pop + p, inv_scale), load_pop_rw<K>(pop + p1, inv_scale));

  // velocities in units of lat_c (1 on the default lattice, where the
  // scalings below are exact)
  V drho, rho, ux, uy, uz;
  if constexpr (GIVEN) {
    const float* r = static_cast<const float*>(a.rho_in);
    const float* u = static_cast<const float*>(a.u_in);
    const float ic = (float)a.lat.ic;
    rho = r[p];
    drho = rho - 1.f;
    ux = u[p] * ic;
    uy = u[a.npad + p] * ic;
    uz = u[2 * a.npad + p] * ic;
  } else {
    macro_vec<V>(f, (float)(0.5 * a.gx), (float)(0.5 * a.gy), (float)(0.5 * a.gz), drho, rho, ux, uy, uz);
  }
  if (WRITE) {
    const V c = VecOf<V>::splat((float)a.lat.c);
    float* u = static_cast<float*>(a.u_out);
    const V cux = vmul(ux, c), cuy = vmul(uy, c), cuz = vmul(uz, c);
#pragma unroll
    for (int j = 0; j < N; j++) {
      const int pj = j == 0 ? p : p1;  // the first node's values again where there is no second
      const int l = both ? j : 0;
      static_cast<float*>(a.rho_out)[pj] = lane(rho, l);
      u[pj] = lane(cux, l);
      u[a.npad + pj] = lane(cuy, l);
      u[2 * a.npad + pj] = lane(cuz, l);
    }
  }
  if (a.snap_dst != nullptr) {
#pragma unroll
    for (int j = 0; j < N; j++) {
      const int pj = j == 0 ? p : second;
      if (pj < a.snap_begin || (j == 1 && !both)) continue;
      double full[kQ];
#pragma unroll
      for (int q = 0; q < kQ; q++) full[q] = to_full<K>(lane(f[q], j), q);
      snap_write(a.snap_dst, a.nsnap, pj - a.snap_begin, full, lane(rho, j), lane(ux, j), lane(uy, j), lane(uz, j));
    }
  }
  collide_vec<V>(f, drho, rho, ux, uy, uz,
                 collide_scalars((float)a.gx, (float)a.gy, (float)a.gz, (float)a.s_v, (float)a.s_o));
  if constexpr (N == 1 || PAIR) {
    store_row<K>(pop + p, f[0], scale, both);
  } else {
    store_pop<K>(pop + p, lane(f[0], 0), scale);
    if (both) store_pop<K>(pop + p1, lane(f[0], 1), scale);
  }
  if constexpr (LOCAL) {
#pragma unroll
    for (int q = 1; q < kQ; q++) store_row<K>(pop + (size_t)q * a.npad + p, f[q], scale, both);
  } else if constexpr (N == 1) {
    for_kept_slots(keep, threadIdx.x, [&](int q, int32_t slot) { store_pop<K>(pop + slot, f[opp(q)], scale); });
  } else {
    for_kept_slots(keep, threadIdx.x, [&](int q, int32_t slot0, int32_t slot1) {
      const float2 v = split_f2(f[opp(q)]);
      store_pop<K>(pop + slot0, v.x, scale);
      if (both) store_pop<K>(pop + slot1, v.y, scale);
    });
  }
}

// Face nodes in deviation storage: the rules act on full populations in
// double, the macro step and collision are the step kernel's.  The slots are
// kept for the stores, as in the step: read from the table again they are 18
// more loads in a row.
template <Store K, int BS, bool GIVEN, bool FINAL>
__global__ void __launch_bounds__(BS, 512 / BS) bc_dev_kernel(BcArgs a) {
  using T = typename Traits<K>::T;
  using A = typename Traits<K>::A;
  using Mac = typename Traits<K>::Mac;
  const int b = blockIdx.x * BS + threadIdx.x;
  const int p = a.s.n_main + b;
  if (p >= a.s.n) return;
  const StepArgs& s = a.s;
  T* pop = static_cast<T*>(s.pop);
  const float scale = (float)s.fp16_scale;
  const float inv_scale = s.fp16_inv;
  __shared__ SlotKeep<FINAL ? 1 : BS, 1> keep;  // slot[q] holds f_q and takes f*_opp(q), in both phases
  double F[kQ];
  {
    int32_t slot[kQ];
#pragma unroll
    for (int q = 1; q < kQ; q++) slot[q] = state_slot(s.phase, s.table, s.npad, p, q);
    F[0] = to_full<K>(load_pop_rw<K>(pop + p, inv_scale), 0);
#pragma unroll
    for (int q = 1; q < kQ; q++) F[q] = to_full<K>(load_pop_rw<K>(pop + slot[q], inv_scale), q);
    if constexpr (!FINAL) keep_slots(keep, threadIdx.x, [&](int q) { return slot[q]; });
  }
  // the rules on the default lattice: velocities here are in units of lat_c
  if (!GIVEN) bc_apply(a, b, F, Lattice{});
  if (FINAL) {
    const size_t nb = (size_t)(s.n - s.n_main);
#pragma unroll
    for (int q = 0; q < kQ; q++) a.bnd_f[(size_t)q * nb + b] = F[q];
    return;
  }
  A f[kQ];
#pragma unroll
  for (int q = 0; q < kQ; q++) f[q] = from_full<K>(F[q], q);
  PairSplit<A> ps;
  split_pairs(f, ps);
  A drho, rho, ux, uy, uz;
  if (GIVEN) {
    const Mac* r = static_cast<const Mac*>(s.rho_in);
    const Mac* u = static_cast<const Mac*>(s.u_in);
    const A ic = A(s.lat.ic);
    rho = (A)r[p];
    drho = rho - A(1);
    ux = (A)u[p] * ic;
    uy = (A)u[s.npad + p] * ic;
    uz = (A)u[2 * s.npad + p] * ic;
  } else {
    if constexpr (sizeof(A) == 4)
      macro_vec<float>(f, (float)(0.5 * s.gx), (float)(0.5 * s.gy), (float)(0.5 * s.gz), drho, rho, ux, uy, uz);
    else
      macro_dev<A>(f, ps, A(0.5 * s.gx), A(0.5 * s.gy), A(0.5 * s.gz), drho, rho, ux, uy, uz);
  }
  if (s.rho_out != nullptr) {
    const A c = A(s.lat.c);
    static_cast<Mac*>(s.rho_out)[p] = (Mac)rho;
    Mac* u = static_cast<Mac*>(s.u_out);
    u[p] = (Mac)(ux * c);
    u[s.npad + p] = (Mac)(uy * c);
    u[2 * s.npad + p] = (Mac)(uz * c);
  }
  snap_write(s.snap_dst, s.nsnap, p - s.snap_begin, F, rho, ux, uy, uz);
  if constexpr (sizeof(A) == 4)
    collide_vec<float>(f, drho, rho, ux, uy, uz,
                       collide_scalars((float)s.gx, (float)s.gy, (float)s.gz, (float)s.s_v, (float)s.s_o));
  else
    mrt_collide_dev<A>(f, ps, drho, rho, ux, uy, uz, A(s.gx), A(s.gy), A(s.gz), A(s.s_v), A(s.s_o));
  store_pop<K>(pop + p, f[0], scale);
  if constexpr (!FINAL)
    for_kept_slots(keep, threadIdx.x, [&](int q, int32_t slot) { store_pop<K>(pop + slot, f[opp(q)], scale); });
}

template <Store K>
static cudaError_t launch_bc_dev(const BcArgs& a, cudaStream_t st) {
  const int nb = a.s.n - a.s.n_main;
  if (nb <= 0) return cudaSuccess;
  auto run = [&](void (*kernel)(BcArgs), int bs) {
    return launch_with(kernel, (nb + bs - 1) / bs, bs, st, false, a.s.carveout, a);
  };
  if (a.bnd_f) return run(bc_dev_kernel<K, 128, false, true>, 128);
  if (a.s.rho_in != nullptr) return run(bc_dev_kernel<K, 128, true, false>, 128);
  switch (face_block(nb)) {
    case 32: return run(bc_dev_kernel<K, 32, false, false>, 32);
    case 64: return run(bc_dev_kernel<K, 64, false, false>, 64);
    default: return run(bc_dev_kernel<K, 128, false, false>, 128);
  }
}

cudaError_t launch_boundary(Store kind, const BcArgs& a, cudaStream_t st) {
  switch (kind) {
    case Store::F64: return launch_boundary_f64(a, st);
    case Store::F64D: return launch_bc_dev<Store::F64D>(a, st);
    case Store::F32: return launch_bc_dev<Store::F32>(a, st);
    case Store::F16: return launch_bc_dev<Store::F16>(a, st);
  }
  return cudaErrorInvalidValue;
}

template <int BS, Slots SL>
static cudaError_t launch_f64d(const StepArgs& a, int grid, cudaStream_t st) {
  const bool given = a.rho_in != nullptr, write = a.rho_out != nullptr;
  if constexpr (SL != Slots::Local) {
    if (given)
      return write ? launch_step_kernel(step_dev_kernel<BS, true, true, SL>, grid, BS, st, a)
                   : launch_step_kernel(step_dev_kernel<BS, true, false, SL>, grid, BS, st, a);
  }
  return write ? launch_step_kernel(step_dev_kernel<BS, false, true, SL>, grid, BS, st, a)
        : launch_step_kernel(step_dev_kernel<BS, false, false, SL>, grid, BS, st, a);
}
template <Store K, int BS, typename V, Slots SL>
static cudaError_t launch_vec(const StepArgs& a, int grid, cudaStream_t st) {
  const bool given = a.rho_in != nullptr, write = a.rho_out != nullptr;
  if constexpr (SL != Slots::Local && VecOf<V>::kNodes == 1) {
    if (given)
      return write ? launch_step_kernel(step_vec_kernel<K, BS, V, true, true, SL>, grid, BS, st, a)
                   : launch_step_kernel(step_vec_kernel<K, BS, V, true, false, SL>, grid, BS, st, a);
  }
  return write ? launch_step_kernel(step_vec_kernel<K, BS, V, false, true, SL>, grid, BS, st, a)
        : launch_step_kernel(step_vec_kernel<K, BS, V, false, false, SL>, grid, BS, st, a);
}

template <Store K, int BS>
static cudaError_t launch_dev_bs(const StepArgs& a, cudaStream_t st) {
  if (a.n_main <= 0) return cudaSuccess;
  const bool local = a.phase == kLocal;
  if (local && a.rho_in != nullptr) return cudaErrorInvalidValue;  // a given state is a kPull state
  const Slots sl = local ? Slots::Local : a.ct_base ? Slots::Compact : Slots::Table;
  const int grid = (a.n_main + BS - 1) / BS;  // BS nodes per block, by BS or BS / 2 threads
  if constexpr (K == Store::F64D) {
    switch (sl) {
      case Slots::Local: return launch_f64d<BS, Slots::Local>(a, grid, st);
      case Slots::Table: return launch_f64d<BS, Slots::Table>(a, grid, st);
      case Slots::Compact: return launch_f64d<BS, Slots::Compact>(a, grid, st);
      default: break;
    }
  } else if (a.rho_in == nullptr && sl != Slots::Compact && two_nodes(a.n_main)) {
    if (local && a.n_main < a.n && (a.n_main & 1)) return launch_vec<K, BS / 2, F2, Slots::LocalOdd>(a, grid, st);
    if (local) return launch_vec<K, BS / 2, F2, Slots::Local>(a, grid, st);
    if constexpr (K == Store::F32)
      if (a.rows) return launch_vec<K, BS / 2, F2, Slots::Rows>(a, grid, st);
    return launch_vec<K, BS / 2, F2, Slots::Table>(a, grid, st);
  } else {
    switch (sl) {
      case Slots::Local: return launch_vec<K, BS, float, Slots::Local>(a, grid, st);
      case Slots::Table: return launch_vec<K, BS, float, Slots::Table>(a, grid, st);
      case Slots::Compact: return launch_vec<K, BS, float, Slots::Compact>(a, grid, st);
      default: break;
    }
  }
  return cudaErrorInvalidValue;
}

template <Store K>
static cudaError_t launch_dev(const StepArgs& a, int block, cudaStream_t st) {
  switch (block) {
    case 64: return launch_dev_bs<K, 64>(a, st);
    case 128: return launch_dev_bs<K, 128>(a, st);
    case 512: return launch_dev_bs<K, 512>(a, st);
    default: return launch_dev_bs<K, 256>(a, st);
  }
}

cudaError_t launch_step(Store kind, const StepArgs& a, int block, cudaStream_t st) {
  switch (kind) {
    case Store::F64: return launch_step_f64(a, block, st);
    case Store::F64D: return launch_dev<Store::F64D>(a, block, st);
    case Store::F32: return launch_dev<Store::F32>(a, block, st);
    case Store::F16: return launch_dev<Store::F16>(a, block, st);
  }
  return cudaErrorInvalidValue;
}

int reduce_blocks(int n) {
  const int b = (n + kReduceThreads - 1) / kReduceThreads;
  return b < 1 ? 1 : (b > 148 * 4 ? 148 * 4 : b);
}

cudaError_t launch_reduce(Store kind, const ReduceArgs& a, cudaStream_t st) {
  switch (kind) {
    case Store::F64: return reduce_f64(a, st);
    case Store::F64D: return reduce_dispatch<Store::F64D>(a, st);
    case Store::F32: return reduce_dispatch<Store::F32>(a, st);
    case Store::F16: return reduce_dispatch<Store::F16>(a, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_export_pop(Store kind, const void* pop, int phase, const int32_t* table, const int32_t* ref_of, int n,
                              int npad, double fp16_scale, double* out, cudaStream_t st, int n_main,
                              const double* bnd_f) {
  switch (kind) {
    case Store::F64: return export_f64(pop, phase, table, ref_of, n, npad, out, st, n_main, bnd_f);
    case Store::F64D:
      return export_dispatch<Store::F64D>(pop, phase, table, ref_of, n, npad, fp16_scale, out, st, n_main, bnd_f);
    case Store::F32:
      return export_dispatch<Store::F32>(pop, phase, table, ref_of, n, npad, fp16_scale, out, st, n_main, bnd_f);
    case Store::F16:
      return export_dispatch<Store::F16>(pop, phase, table, ref_of, n, npad, fp16_scale, out, st, n_main, bnd_f);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_import_pop(Store kind, void* pop, const int32_t* table, const int32_t* ref_of, int n, int npad,
                              double fp16_scale, const double* in, cudaStream_t st) {
  switch (kind) {
    case Store::F64: return import_f64(pop, table, ref_of, n, npad, in, st);
    case Store::F64D: return import_dispatch<Store::F64D>(pop, table, ref_of, n, npad, fp16_scale, in, st);
    case Store::F32: return import_dispatch<Store::F32>(pop, table, ref_of, n, npad, fp16_scale, in, st);
    case Store::F16: return import_dispatch<Store::F16>(pop, table, ref_of, n, npad, fp16_scale, in, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_import_macro(Store kind, void* rho, void* u, const int32_t* ref_of, int n, int npad,
                                const double* rho_in, const double* u_in, cudaStream_t st) {
  switch (kind) {
    case Store::F64: return import_macro_f64(rho, u, ref_of, n, npad, rho_in, u_in, st);
    case Store::F64D: return import_macro_dispatch<Store::F64D>(rho, u, ref_of, n, npad, rho_in, u_in, st);
    case Store::F32: return import_macro_dispatch<Store::F32>(rho, u, ref_of, n, npad, rho_in, u_in, st);
    case Store::F16: return import_macro_dispatch<Store::F16>(rho, u, ref_of, n, npad, rho_in, u_in, st);
  }
  return cudaErrorInvalidValue;
}

__global__ void export_macro_kernel(const double* __restrict__ rho_int, const double* __restrict__ u_int,
                                    const int32_t* __restrict__ ref_of, int n, int npad, double* __restrict__ rho_ref,
                                    double* __restrict__ u_ref) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int r = ref_of[p];
  if (rho_ref) rho_ref[r] = rho_int[p];
  if (u_ref) {
    u_ref[(size_t)r * 3 + 0] = u_int[p];
    u_ref[(size_t)r * 3 + 1] = u_int[npad + p];
    u_ref[(size_t)r * 3 + 2] = u_int[2 * npad + p];
  }
}

cudaError_t launch_export_macro(const double* rho_int, const double* u_int, const int32_t* ref_of, int n, int npad,
                                double* rho_ref, double* u_ref, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  export_macro_kernel<<<(n + 255) / 256, 256, 0, st>>>(rho_int, u_int, ref_of, n, npad, rho_ref, u_ref);
  return cudaGetLastError();
}

// One scalar field in the reference's order, row 0 zero.
template <typename T>
__global__ void export_scalar_kernel(const T* __restrict__ src, const int32_t* __restrict__ ref_of, int n,
                                     double* __restrict__ out) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p == 0) out[0] = 0.0;
  if (p < n) out[ref_of[p]] = (double)src[p];
}

cudaError_t launch_export_scalar(bool f64, const void* src, const int32_t* ref_of, int n, double* out,
                                 cudaStream_t st) {
  const int g = n > 0 ? (n + 255) / 256 : 1;
  if (f64)
    export_scalar_kernel<<<g, 256, 0, st>>>(static_cast<const double*>(src), ref_of, n, out);
  else
    export_scalar_kernel<<<g, 256, 0, st>>>(static_cast<const float*>(src), ref_of, n, out);
  return cudaGetLastError();
}

struct Feq19 {
  double v[kQ];
};

template <Store K>
__global__ void init_uniform_kernel(typename Traits<K>::T* __restrict__ pop, const int32_t* __restrict__ table, int n,
                                    int npad, float scale, Feq19 feq) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  store_pop<K>(pop + p, from_full<K>(feq.v[0], 0), scale);
#pragma unroll
  for (int q = 1; q < kQ; q++)
    store_pop<K>(pop + table[(size_t)(q - 1) * npad + p], from_full<K>(feq.v[q], q), scale);
}

template <typename Mac>
__global__ void fill_macro_kernel(Mac* __restrict__ rho, Mac* __restrict__ u, int n, int npad, double rho0,
                                  double ux, double uy, double uz) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  rho[p] = (Mac)rho0;
  u[p] = (Mac)ux;
  u[npad + p] = (Mac)uy;
  u[2 * npad + p] = (Mac)uz;
}

cudaError_t launch_init_uniform(Store kind, void* pop, const int32_t* table, int n, int npad, double fp16_scale,
                                const double* feq19, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  Feq19 f;
  for (int q = 0; q < kQ; q++) f.v[q] = feq19[q];
  const int g = (n + 255) / 256;
  const float sc = (float)fp16_scale;
  switch (kind) {
    case Store::F64: init_uniform_kernel<Store::F64><<<g, 256, 0, st>>>((double*)pop, table, n, npad, sc, f); break;
    case Store::F64D: init_uniform_kernel<Store::F64D><<<g, 256, 0, st>>>((double*)pop, table, n, npad, sc, f); break;
    case Store::F32: init_uniform_kernel<Store::F32><<<g, 256, 0, st>>>((float*)pop, table, n, npad, sc, f); break;
    case Store::F16: init_uniform_kernel<Store::F16><<<g, 256, 0, st>>>((__half*)pop, table, n, npad, sc, f); break;
  }
  return cudaGetLastError();
}

cudaError_t launch_fill_macro(Store kind, void* rho, void* u, int n, int npad, double rho0, const double* u3,
                              cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const int g = (n + 255) / 256;
  if (kind == Store::F64 || kind == Store::F64D)
    fill_macro_kernel<double><<<g, 256, 0, st>>>((double*)rho, (double*)u, n, npad, rho0, u3[0], u3[1], u3[2]);
  else
    fill_macro_kernel<float><<<g, 256, 0, st>>>((float*)rho, (float*)u, n, npad, rho0, u3[0], u3[1], u3[2]);
  return cudaGetLastError();
}

size_t store_bytes(Store kind) {
  switch (kind) {
    case Store::F64:
    case Store::F64D: return 8;
    case Store::F32: return 4;
    case Store::F16: return 2;
  }
  return 8;
}

}  // namespace lbm
