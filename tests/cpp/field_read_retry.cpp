// A field read that runs out of device memory reports it, touches no memory,
// and the next read gives the plain read's values.
//
// The solvers' host code runs here on a CUDA runtime of host memory: device
// buffers are host allocations kept in a table, every launcher of the field
// reads checks that what it is given lies inside one of them before it writes,
// and the n-th device allocation from now can be made to fail.  As CUDA does,
// a failed call leaves its code for the next cudaGetLastError.
#include "fake_cuda.h"

#include "batch.h"
#include "cg_api.h"
#include "setup.h"
#include "st7_api.h"

using namespace lbm;

// ---------------------------------------------------------- launchers
namespace lbm {
size_t store_bytes(Store k) { return k == Store::F16 ? 2 : k == Store::F32 ? 4 : 8; }
int reduce_blocks(int) { return 1; }
int batch_step_grid(int ntiles, int) { return ntiles; }
cudaError_t launch_init_uniform(Store, void*, const int32_t*, int, int, double, const double*, cudaStream_t) {
  return last();
}
cudaError_t launch_row_table(const int32_t*, int, int, int32_t*, int*, cudaStream_t) { return last(); }
void SetupScratch::release() {}
lbm_status device_index_reference(const uint8_t*, int, int, int, int, int32_t*, long long, int, int32_t*,
                                  SetupScratch&, cudaStream_t) {
  return LBM_OK;
}
cudaError_t launch_export_macro(const double* r, const double* u, const int32_t* ref_of, int n, int npad, double* rr,
                                double* ur, cudaStream_t) {
  need(r, sizeof(double) * npad, "internal rho");
  need(u, sizeof(double) * 3 * npad, "internal u");
  need(rr, sizeof(double) * (n + 1), "rho");
  need(ur, sizeof(double) * 3 * (n + 1), "u");
  for (int p = 0; p < n; p++) {
    rr[ref_of[p]] = r[p];
    for (int d = 0; d < 3; d++) ur[3 * ref_of[p] + d] = u[(size_t)d * npad + p];
  }
  return last();
}
cudaError_t launch_export_scalar(bool f64, const void* src, const int32_t* ref_of, int n, double* out, cudaStream_t) {
  need(src, (f64 ? 8 : 4) * (size_t)n, "scalar field");
  need(out, sizeof(double) * (n + 1), "scalar field out");
  out[0] = 0.0;
  for (int p = 0; p < n; p++)
    out[ref_of[p]] = f64 ? static_cast<const double*>(src)[p] : (double)static_cast<const float*>(src)[p];
  return last();
}
// two-phase
cudaError_t cg_set_mi_f64(const double*, cudaStream_t) { return last(); }
cudaError_t cg_set_mi_f32(const double*, cudaStream_t) { return last(); }
bool cg_block_pattern_matches(const double*) { return true; }
cudaError_t cg_colour_f64(const CgArgs&, cudaStream_t) { return last(); }
cudaError_t cg_colour_f32(const CgArgs&, cudaStream_t) { return last(); }
static cudaError_t cg_reduce(const CgReduceArgs& a) {
  need(a.rho_out, sizeof(double) * a.npad, "two-phase rho");
  need(a.u_out, sizeof(double) * 3 * a.npad, "two-phase u");
  for (int p = 0; p < a.n; p++) {
    a.rho_out[p] = 100 + p;
    for (int d = 0; d < 3; d++) a.u_out[(size_t)d * a.npad + p] = 1000 * (d + 1) + p;
  }
  return last();
}
cudaError_t cg_reduce_f64(const CgReduceArgs& a, int, cudaStream_t) { return cg_reduce(a); }
cudaError_t cg_reduce_f32(const CgReduceArgs& a, int, cudaStream_t) { return cg_reduce(a); }
// solute
cudaError_t st7_launch_init(bool, const St7Args&, cudaStream_t) { return last(); }
cudaError_t st7_launch_conc(bool, const St7Args& a, double* out, cudaStream_t) {
  need(out, sizeof(double) * a.n, "concentration");
  for (int p = 0; p < a.n; p++) out[p] = 7 + p;
  return last();
}
// node pool
cudaError_t launch_batch_init(Store, void*, int, const int32_t*, int, int, int, const InstParams&, cudaStream_t) {
  return last();
}
cudaError_t launch_batch_export_macro(Store, const void*, int, const int32_t*, int, int, int n, const int32_t*,
                                      const InstParams&, double* rho, double* u, cudaStream_t) {
  need(rho, sizeof(double) * (n + 1), "pool rho");
  need(u, sizeof(double) * 3 * (n + 1), "pool u");
  for (int p = 1; p <= n; p++) {
    rho[p] = 50 + p;
    for (int d = 0; d < 3; d++) u[3 * p + d] = d * 10 + p;
  }
  return last();
}
}  // namespace lbm

// ---------------------------------------------------------------- test
static void check(bool ok, const char* what) {
  if (ok) return;
  std::printf("failed: %s (%s)\n", what, lbm_last_error());
  std::exit(1);
}

// read(values) is the field read; every device allocation it makes is failed
// in turn, on the first read of a new handle, and the read made again.
template <typename Create, typename Read, typename Destroy>
static void retry(const char* name, size_t nvalues, Create create, Read read, Destroy destroy) {
  std::vector<double> plain(nvalues, -1.0), again(nvalues);
  {
    auto* h = create();
    check(read(h, plain.data()) == LBM_OK, name);
    destroy(h);
  }
  int failures = 0;
  for (int k = 1;; k++) {
    auto* h = create();
    g_fail_in = k;
    const lbm_status st = read(h, again.data());
    const bool reached = g_fail_in == 0;
    g_fail_in = 0;
    if (reached) {
      failures++;
      check(st == LBM_ERR_OOM, name);
      again.assign(nvalues, -1.0);
      check(read(h, again.data()) == LBM_OK, name);
    } else {
      check(st == LBM_OK, name);
    }
    check(again == plain, name);
    destroy(h);
    if (!reached) break;
  }
  check(failures > 0, "the read allocates");
}

// Every subset of the five two-phase fields is the plain read's values.
static void subsets(lbm_cg_handle* h, size_t r) {
  std::vector<double> all(7 * r);
  const size_t at[5] = {0, r, 4 * r, 5 * r, 6 * r}, len[5] = {r, 3 * r, r, r, r};
  check(lbm_cg_get_fields(h, &all[0], &all[r], &all[4 * r], &all[5 * r], &all[6 * r]) == LBM_OK, "all fields");
  for (int m = 0; m < 32; m++) {
    std::vector<double> v(7 * r, -1.0);
    double* p[5];
    for (int i = 0; i < 5; i++) p[i] = (m >> i & 1) ? &v[at[i]] : nullptr;
    check(lbm_cg_get_fields(h, p[0], p[1], p[2], p[3], p[4]) == LBM_OK, "some fields");
    for (int i = 0; i < 5; i++)
      for (size_t k = 0; k < len[i]; k++)
        check(v[at[i] + k] == ((m >> i & 1) ? all[at[i] + k] : -1.0), "values of some fields");
  }
}

int main(int argc, char** argv) {
  g_fail_pin = argc > 1 && !std::strcmp(argv[1], "nopin");
  const int nx = 9, ny = 7, nz = 6;
  std::vector<uint8_t> mask(nx * ny * nz, 0);
  std::vector<double> psi(mask.size());
  size_t n = 0;
  for (size_t i = 0; i < mask.size(); i++) {
    mask[i] = (i * 7) % 5 == 0;
    psi[i] = mask[i] ? 0.0 : (i % 2 ? 1.0 : -1.0);
    n += !mask[i];
  }
  const size_t r = n + 1;
  for (int precision : {LBM_PREC_F64, LBM_PREC_F32}) {
    retry(
        "two-phase fields", 7 * r,
        [&] {
          lbm_cg_params p{};
          p.nu_l = p.nu_g = 0.1;
          p.psi_solid = 0.7;
          p.cap_a = 1e-3;
          p.perdir = 1;
          p.precision = precision;
          lbm_cg_handle* h = nullptr;
          check(lbm_cg_create(&p, mask.data(), psi.data(), nx, ny, nz, &h) == LBM_OK, "lbm_cg_create");
          return h;
        },
        [&](lbm_cg_handle* h, double* v) {
          return lbm_cg_get_fields(h, v, v + r, v + 4 * r, v + 5 * r, v + 6 * r);
        },
        lbm_cg_destroy);
    {
      lbm_cg_params p{};
      p.nu_l = p.nu_g = 0.1;
      p.psi_solid = 0.7;
      p.cap_a = 1e-3;
      p.perdir = 1;
      p.precision = precision;
      lbm_cg_handle* h = nullptr;
      check(lbm_cg_create(&p, mask.data(), psi.data(), nx, ny, nz, &h) == LBM_OK, "lbm_cg_create");
      subsets(h, r);
      lbm_cg_destroy(h);
    }
    for (int lattice : {7, 19})
      retry(
          "solute concentration", r,
          [&] {
            lbm_st7_params p{};
            p.diffusivity = 0.01;
            p.precision = precision;
            std::vector<double> c0(mask.size(), 0.5), u(3 * r, 0.0);
            lbm_st7_handle* h = nullptr;
            const auto create = lattice == 7 ? lbm_st7_create : lbm_st19_create;
            check(create(&p, mask.data(), nx, ny, nz, u.data(), c0.data(), &h) == LBM_OK, "solute create");
            return h;
          },
          [&](lbm_st7_handle* h, double* v) { return lbm_st7_get_concentration(h, v); }, lbm_st7_destroy);
  }
  retry(
      "pool fields", 4 * r,
      [&] {
        lbm_instance in{};
        in.mask = mask.data();
        in.nx = nx;
        in.ny = ny;
        in.nz = nz;
        in.nu = 0.1;
        in.gx = 1e-6;
        lbm_batch* b = nullptr;
        check(lbm_batch_create(1, &in, LBM_PREC_F32, LBM_ORDER_REFERENCE, 512, 0, &b) == LBM_OK, "lbm_batch_create");
        return b;
      },
      [&](lbm_batch* b, double* v) { return lbm_batch_get_fields(b, 0, v, v + r); }, lbm_batch_destroy);
  std::printf("ok\n");
  return 0;
}
