// How the steps of a call reach the device: captured chains of 16 steps or
// single launches, for calls of every length (no GPU; fake_cuda.h).
#include "fake_cuda.h"

#include "lbm_internal.h"
#include "setup.h"
#include "st7_api.h"

using namespace lbm;

static int g_steps = 0;  // launched outside captures

namespace lbm {
size_t store_bytes(Store k) { return k == Store::F16 ? 2 : k == Store::F32 ? 4 : 8; }
int reduce_blocks(int) { return 1; }
bool mi_pattern_matches(const double*) { return true; }
cudaError_t set_mi_constant(const double*, cudaStream_t) { return last(); }
cudaError_t launch_init_uniform(Store, void*, const int32_t*, int, int, double, const double*, cudaStream_t) {
  return last();
}
cudaError_t launch_fill_macro(Store, void*, void*, int, int, double, const double*, cudaStream_t) { return last(); }
cudaError_t launch_row_table(const int32_t*, int, int, int32_t*, int*, cudaStream_t) { return last(); }
bool SetupScratch::borrow(void*, size_t, long long, int) { return true; }
void SetupScratch::release() {}
lbm_status device_index_reference(const uint8_t*, int, int, int, int, int32_t*, long long, int, int32_t*,
                                  SetupScratch&, cudaStream_t) {
  return LBM_OK;
}
cudaError_t launch_step(Store, const StepArgs& a, int, cudaStream_t) {
  if (!g_capturing) g_steps++;
  // a given state is a kPull state, and the phase is the one of a step chain
  if (a.rho_in != nullptr && a.phase == kLocal) return cudaErrorInvalidValue;
  return last();
}
cudaError_t st7_launch_init(bool, const St7Args&, cudaStream_t) { return last(); }
cudaError_t st7_launch_step(bool, const St7Args& a, cudaStream_t) {
  if (!g_capturing) g_steps++;
  if (a.c_given != nullptr && a.phase == kLocal) return cudaErrorInvalidValue;
  return last();
}
}  // namespace lbm

static void check(bool ok, const char* what, long long a = 0, long long b = 0) {
  if (ok) return;
  std::printf("failed: %s (%lld, %lld) %s\n", what, a, b, lbm_last_error());
  std::exit(1);
}

int main(int argc, char** argv) {
  const int nx = 9, ny = 7, nz = 6;
  std::vector<uint8_t> mask(nx * ny * nz, 0);
  for (size_t i = 0; i < mask.size(); i += 5) mask[i] = 1;
  size_t n = 0;
  for (uint8_t m : mask) n += !m;
  if (argc > 1 && argv[1][0] == 'f') {
    for (int k = 1; k <= 67; k++) {
      lbm_params p;
      lbm_params_default(&p);
      lbm_handle* h = nullptr;
      check(lbm_create(&p, mask.data(), nx, ny, nz, &h) == LBM_OK, "lbm_create");
      g_captures = g_replays = g_steps = 0;
      const int calls = 40;
      int before = 0, replays = 0;
      for (int c = 0; c < calls; c++) {
        before = g_steps;
        replays = g_replays;
        check(lbm_step(h, k) == LBM_OK, "lbm_step", k);
        check(16 * (g_replays - replays) + g_steps - before == k, "steps of a call", k, c);
        // one chain is captured for the first call, the other only for calls that need it
        if (c == 0) check(g_captures == (k >= 19), "chains captured by the first call", k, g_captures);
        // a call that a chain fits in goes through chains, all but its last step and the rest of 16
        if (c >= calls / 2) check(g_steps - before <= 1 + (k - 1) % 16, "single steps", k, g_steps - before);
      }
      long long step = 0;
      check(lbm_info(h, nullptr, nullptr, &step) == LBM_OK && step == (long long)calls * k, "step counter", k, step);
      lbm_destroy(h);
    }
  } else {
    std::vector<double> c0(mask.size(), 0.5), u(3 * (n + 1), 0.0);
    for (int k = 1; k <= 300; k++) {
      lbm_st7_params p{};
      p.diffusivity = 0.01;
      lbm_st7_handle* h = nullptr;
      check(lbm_st7_create(&p, mask.data(), nx, ny, nz, u.data(), c0.data(), &h) == LBM_OK, "lbm_st7_create");
      g_captures = g_replays = g_steps = 0;
      check(lbm_st7_step(h, k) == LBM_OK, "lbm_st7_step", k);
      check(16 * g_replays + g_steps == k, "steps of the first call", k);
      // a first call captures what it replays, and nothing for a few steps
      check(g_captures == (k > 128), "chains captured by the first call", k, g_captures);
      for (int c = 0; c < 40; c++) {
        const int before = g_steps;
        check(lbm_st7_step(h, k) == LBM_OK, "lbm_st7_step", k);
        if (c >= 20) check(g_steps - before <= k % 16, "single steps", k, g_steps - before);
      }
      check(g_captures <= 2, "chains captured", k, g_captures);
      lbm_st7_destroy(h);
    }
  }
  std::printf("ok\n");
  return 0;
}
