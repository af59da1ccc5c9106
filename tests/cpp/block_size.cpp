// The block size that reaches the step's launch: the one asked for, the
// solver's own choice where none was, and the ones the autotuners time (no
// GPU; fake_cuda.h).
#include "fake_cuda.h"

#include <set>

#include "batch.h"
#include "lbm_internal.h"
#include "setup.h"

using namespace lbm;

static std::vector<int> g_blocks;  // of every step launched or captured

namespace lbm {
size_t store_bytes(Store k) { return k == Store::F16 ? 2 : k == Store::F32 ? 4 : 8; }
int reduce_blocks(int) { return 1; }
int batch_step_grid(int ntiles, int) { return ntiles; }
bool mi_pattern_matches(const double*) { return true; }
cudaError_t set_mi_constant(const double*, cudaStream_t) { return last(); }
cudaError_t launch_init_uniform(Store, void*, const int32_t*, int, int, double, const double*, cudaStream_t) {
  return last();
}
cudaError_t launch_fill_macro(Store, void*, void*, int, int, double, const double*, cudaStream_t) { return last(); }
cudaError_t launch_row_table(const int32_t*, int, int, int32_t*, int*, cudaStream_t) { return last(); }
cudaError_t launch_compact_table(const int32_t*, int, int, int32_t*, uint16_t*, unsigned long long*, cudaStream_t) {
  return last();
}
cudaError_t launch_export_pop(Store, const void*, int, const int32_t*, const int32_t*, int, int, double, double*,
                              cudaStream_t, int, const double*) {
  return last();
}
cudaError_t launch_import_pop(Store, void*, const int32_t*, const int32_t*, int, int, double, const double*,
                              cudaStream_t) {
  return last();
}
cudaError_t launch_import_macro(Store, void*, void*, const int32_t*, int, int, const double*, const double*,
                                cudaStream_t) {
  return last();
}
cudaError_t launch_export_macro(const double*, const double*, const int32_t*, int, int, double*, double*,
                                cudaStream_t) {
  return last();
}
cudaError_t launch_reduce(Store, const ReduceArgs&, cudaStream_t) { return last(); }
bool SetupScratch::borrow(void*, size_t, long long, int) { return true; }
void SetupScratch::release() {}
lbm_status device_index_reference(const uint8_t*, int, int, int, int, int32_t*, long long, int, int32_t*,
                                  SetupScratch&, cudaStream_t) {
  return LBM_OK;
}
cudaError_t launch_step(Store, const StepArgs&, int block, cudaStream_t) {
  g_blocks.push_back(block);
  return last();
}
cudaError_t launch_batch_init(Store, void*, int, const int32_t*, int, int, int, const InstParams&, cudaStream_t) {
  return last();
}
cudaError_t launch_batch_list(const BatchReduceArgs&, int, int, cudaStream_t) { return last(); }
cudaError_t launch_batch_step(Store, const BatchStepArgs&, int block, int, int, cudaStream_t) {
  g_blocks.push_back(block);
  return last();
}
// captured once per chain graph: ends all solves but the first g_keep
static int g_keep = 0;
cudaError_t launch_batch_check(Store, const BatchReduceArgs& a, int, double, long long, cudaStream_t) {
  for (int i = g_keep; i < a.nslots; i++) a.state[i].active = 0, a.state[i].done = 1;
  g_keep = 0;
  return last();
}
}  // namespace lbm

static void check(bool ok, const char* what, long long a = 0, long long b = 0) {
  if (ok) return;
  std::printf("failed: %s (%lld, %lld) %s\n", what, a, b, lbm_last_error());
  std::exit(1);
}

int main() {
  const int nx = 40, ny = 30, nz = 30;
  std::vector<uint8_t> mask(nx * ny * nz, 0);
  const size_t nodes = mask.size();
  for (int precision : {LBM_PREC_F64, LBM_PREC_F32, LBM_PREC_F16, LBM_PREC_F64_FAST})
    for (int block : {0, 64, 128, 256, 512}) {
      lbm_params p;
      lbm_params_default(&p);
      check(p.block_size == 0, "the default asks for no size");
      p.precision = precision;
      p.block_size = block;
      lbm_handle* h = nullptr;
      check(lbm_create(&p, mask.data(), nx, ny, nz, &h) == LBM_OK, "lbm_create");
      g_blocks.clear();
      check(lbm_step(h, 40) == LBM_OK, "lbm_step");
      const Store k = precision == LBM_PREC_F64 ? Store::F64
                      : precision == LBM_PREC_F64_FAST ? Store::F64D
                      : precision == LBM_PREC_F32 ? Store::F32 : Store::F16;
      for (int b : g_blocks) check(b == (block ? block : default_block(k, nodes)), "flow block", block, b);
      if (block == 0) {
        int order = 0, best = 0;
        double ml = 0;
        g_blocks.clear();
        check(lbm_autotune(h, 4, &order, &best, &ml) == LBM_OK, "lbm_autotune");
        const std::set<int> tried(g_blocks.begin(), g_blocks.end());
        check(tried == std::set<int>({64, 128, 256, 512}), "sizes the autotuner times");
        check(tried.count(best) == 1, "the size it reports", best);
        g_blocks.clear();
        check(lbm_step(h, 40) == LBM_OK, "lbm_step");
        for (int b : g_blocks) check(b == best, "block after autotuning", best, b);
      }
      lbm_destroy(h);
    }
  lbm_instance in{};
  in.mask = mask.data();
  in.nx = nx;
  in.ny = ny;
  in.nz = nz;
  in.nu = 0.1;
  in.gx = 1e-6;
  for (int count : {1, 8})  // 71 tiles, a grid of 128; 568 tiles, a grid of 568
    for (int block : {-1, 128, 256, 512}) {
      const std::vector<lbm_instance> all(count, in);
      lbm_batch* b = nullptr;
      check(lbm_batch_create(count, all.data(), LBM_PREC_F32, LBM_ORDER_REFERENCE, block, 0, &b) == LBM_OK,
            "lbm_batch_create");
      g_blocks.clear();
      check(lbm_batch_run(b, 1e-6, 10, 1000, nullptr) == LBM_OK, "lbm_batch_run");
      check(!g_blocks.empty(), "pool steps");
      for (int s : g_blocks) check(s == (block > 0 ? block : count == 1 ? 512 : 256), "pool block", block, s);
      if (block == -1) {
        int order = 0, best = 0;
        double ml = 0;
        g_blocks.clear();
        check(lbm_batch_autotune(b, 4, &order, &best, &ml) == LBM_OK, "lbm_batch_autotune");
        const std::set<int> tried(g_blocks.begin(), g_blocks.end());
        check(tried == std::set<int>({128, 256, 512}) && tried.count(best) == 1, "sizes the pool's autotuner times", best);
        g_blocks.clear();
        check(lbm_batch_run(b, 1e-6, 10, 1000, nullptr) == LBM_OK, "lbm_batch_run");
        for (int s : g_blocks) check(s == best, "pool block after autotuning", best, s);
        if (count == 8) {  // 568 tiles, then the 71 of the solve that is left
          check(best == 128, "equal times: the first size", best);
          check(lbm_batch_autotune(b, 4, &order, &best, &ml) == LBM_OK, "lbm_batch_autotune");
          g_blocks.clear();
          g_keep = 1;
          check(lbm_batch_run(b, 1e-6, 10, 1000, nullptr) == LBM_OK, "lbm_batch_run");
          check(g_blocks.size() == 20, "two chains", g_blocks.size());
          for (size_t i = 0; i < g_blocks.size(); i++)
            check(g_blocks[i] == (i < 10 ? best : 512), "tuned block as solves stop", i, g_blocks[i]);
        }
      }
      lbm_batch_destroy(b);
    }
  std::printf("ok\n");
  return 0;
}
