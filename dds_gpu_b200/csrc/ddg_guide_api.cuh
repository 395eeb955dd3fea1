// C ABI of the learned guide (include/ddg.h, ddg_guide_*): parameters, one training step
// (forward, loss, backward and Adam, all on the GPU in this file's kernels) and inference
// of NS seeds and root leads. Included at the end of ddg_api.cu.
#pragma once
#include "ddg_guide.cuh"

struct ddg_guide {
  int device = 0;
  int max_rows = 0;
  long long step = 0;
  float* master = nullptr;  // fp32 parameters (flat layout of guide_nn::N_PARAMS)
  float* adam_m = nullptr;
  float* adam_v = nullptr;
  float* grad = nullptr;
  unsigned char* packed = nullptr;  // bf16 weights in the tensor cores' layout (guide_nn::PK_*)
  // a training step's workspace for max_rows rows, [column][row]
  guide_nn::bf16 *Xt = nullptr, *H1t = nullptr, *H2t = nullptr, *dOt = nullptr, *dZ1t = nullptr, *dZ2t = nullptr;
  float *Z1t = nullptr, *Z2t = nullptr;
  float* part = nullptr;  // weight-gradient parts: splits x 5 x 128 x 256
  float* acc = nullptr;   // loss, hits, rows, and the error flag behind them
  int64_t* rows_buf = nullptr;
  int* err = nullptr;  // = acc + 3
  int sms = 0;
};

namespace guide_nn {

static bool g_attr_done[64];

static int set_kernel_attrs() {
  int dev = 0;
  CUDA_TRY(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && g_attr_done[dev]) return DDG_OK;
  CUDA_TRY(cudaFuncSetAttribute((const void*)mlp_rows<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, MLP_SMEM));
  CUDA_TRY(cudaFuncSetAttribute((const void*)mlp_rows<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, MLP_SMEM));
  CUDA_TRY(cudaFuncSetAttribute((const void*)gemm_dw, cudaFuncAttributeMaxDynamicSharedMemorySize, DW_SMEM));
  if (dev >= 0 && dev < 64) g_attr_done[dev] = true;
  return DDG_OK;
}

// Batch rows to a split of the weight gradients (a multiple of 128), at most 32 splits.
static int dw_rows(int R) { return (R / DW_K + 31) / 32 * DW_K; }
static int dw_splits(int R) { return (R + dw_rows(R) - 1) / dw_rows(R); }

static int refresh_packed(ddg_guide* g, cudaStream_t st) {
  pack_params<<<((int)N_PARAMS + 255) / 256, 256, 0, st>>>(g->master, g->packed);
  CUDA_TRY(cudaGetLastError());
  return DDG_OK;
}

static int check_err(ddg_guide* g) {
  int e = 0;
  CUDA_TRY(cudaMemcpy(&e, g->err, 4, cudaMemcpyDeviceToHost));
  if (e) return fail(DDG_E_TIMEOUT, "guide: a tensor-core product did not complete (bounded wait)");
  return DDG_OK;
}

}  // namespace guide_nn

extern "C" {

int64_t ddg_guide_param_count(void) { return guide_nn::N_PARAMS; }

void ddg_guide_destroy(ddg_guide* g) {
  if (!g) return;
  cudaSetDevice(g->device);
  void* bufs[] = {g->master, g->adam_m, g->adam_v, g->grad, g->packed, g->Xt, g->H1t, g->H2t, g->dOt, g->dZ1t, g->dZ2t,
                  g->Z1t, g->Z2t, g->part, g->acc, g->rows_buf};
  for (void* b : bufs) cudaFree(b);
  delete g;
}

int ddg_guide_create(int device, int max_rows, const float* params, ddg_guide** out) {
  using namespace guide_nn;
  if (!out) return fail(DDG_E_ARG, "null output");
  *out = nullptr;
  if (max_rows <= 0 || max_rows % TILE_M || max_rows > (1 << 20))
    return fail(DDG_E_ARG, "max_rows %d is not a positive multiple of 128 (<= 1M)", max_rows);
  CUDA_TRY(cudaSetDevice(device));
  int rc = set_kernel_attrs();
  if (rc) return rc;
  ddg_guide* g = new ddg_guide();
  g->device = device;
  g->max_rows = max_rows;
  const size_t R = (size_t)max_rows, P = (size_t)N_PARAMS;
  cudaError_t e = cudaSuccess;
  auto A = [&](void** p, size_t bytes) {
    if (e == cudaSuccess) e = cudaMalloc(p, bytes);
    if (e == cudaSuccess) e = cudaMemset(*p, 0, bytes);
  };
  A((void**)&g->master, P * 4);
  A((void**)&g->adam_m, P * 4);
  A((void**)&g->adam_v, P * 4);
  A((void**)&g->grad, P * 4);
  A((void**)&g->packed, PK_BYTES);
  A((void**)&g->Xt, R * IN_PAD * 2);
  A((void**)&g->H1t, R * HID * 2);
  A((void**)&g->H2t, R * HID * 2);
  A((void**)&g->dOt, R * DO_LD * 2);
  A((void**)&g->dZ1t, R * HID * 2);
  A((void**)&g->dZ2t, R * HID * 2);
  A((void**)&g->Z1t, R * HID * 4);
  A((void**)&g->Z2t, R * HID * 4);
  // (the splits of any step's rows: at most 32, and a step of fewer rows may have more than the largest)
  A((void**)&g->part, (size_t)std::min(32, max_rows / DW_K) * DW_TILES * TILE_M * HID * 4);
  A((void**)&g->acc, 4 * 4);
  A((void**)&g->rows_buf, R * 8);
  g->err = reinterpret_cast<int*>(g->acc + 3);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&g->sms, cudaDevAttrMultiProcessorCount, device);
  if (e == cudaSuccess && params) e = cudaMemcpy(g->master, params, P * 4, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    ddg_guide_destroy(g);
    return fail(e == cudaErrorMemoryAllocation ? DDG_E_MEMORY : DDG_E_CUDA, "guide buffers: %s",
                cudaGetErrorString(e));
  }
  rc = refresh_packed(g, nullptr);
  if (rc == DDG_OK && cudaDeviceSynchronize() != cudaSuccess) rc = fail(DDG_E_CUDA, "guide init");
  if (rc) {
    ddg_guide_destroy(g);
    return rc;
  }
  *out = g;
  return DDG_OK;
}

int ddg_guide_get_params(ddg_guide* g, float* params) {
  if (!g || !params) return fail(DDG_E_ARG, "null argument");
  CUDA_TRY(cudaSetDevice(g->device));
  CUDA_TRY(cudaMemcpy(params, g->master, guide_nn::N_PARAMS * 4, cudaMemcpyDeviceToHost));
  return DDG_OK;
}

int ddg_guide_set_params(ddg_guide* g, const float* params) {
  if (!g || !params) return fail(DDG_E_ARG, "null argument");
  CUDA_TRY(cudaSetDevice(g->device));
  CUDA_TRY(cudaMemcpy(g->master, params, guide_nn::N_PARAMS * 4, cudaMemcpyHostToDevice));
  int rc = guide_nn::refresh_packed(g, nullptr);
  if (rc) return rc;
  CUDA_TRY(cudaDeviceSynchronize());
  return DDG_OK;
}

int ddg_guide_train_step(ddg_guide* g, const uint64_t* d_hands, const uint8_t* d_tricks20, const int8_t* d_best20,
                         const int64_t* rows_host, int n_rows, float lr, float* stats3, float* grad_host) {
  using namespace guide_nn;
  if (!g || !d_hands || !d_tricks20 || !d_best20 || !rows_host) return fail(DDG_E_ARG, "null argument");
  if (n_rows <= 0 || n_rows > g->max_rows) return fail(DDG_E_ARG, "%d rows (max %d)", n_rows, g->max_rows);
  CUDA_TRY(cudaSetDevice(g->device));
  const int R = (n_rows + TILE_M - 1) / TILE_M * TILE_M;  // padded rows carry no example
  std::vector<int64_t> rows(R, -1);
  for (int i = 0; i < n_rows; i++) rows[i] = rows_host[i];
  cudaStream_t st = nullptr;
  CUDA_TRY(cudaMemcpy(g->rows_buf, rows.data(), (size_t)R * 8, cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMemsetAsync(g->acc, 0, 16, st));  // the sums and the error flag
  MlpArgs a;
  memset(&a, 0, sizeof(a));
  a.hands = d_hands;
  a.rows = g->rows_buf;
  a.n = a.R = R;
  a.tiles = R / TILE_M;
  a.packed = g->packed;
  a.master = g->master;
  a.tricks20 = d_tricks20;
  a.best20 = d_best20;
  a.Xt = g->Xt;
  a.H1t = g->H1t;
  a.H2t = g->H2t;
  a.dOt = g->dOt;
  a.dZ2t = g->dZ2t;
  a.dZ1t = g->dZ1t;
  a.Z1t = g->Z1t;
  a.Z2t = g->Z2t;
  a.acc = g->acc;
  a.err = g->err;
  mlp_rows<true><<<std::min(a.tiles, g->sms), MLP_THREADS<true>, MLP_SMEM, st>>>(a);
  const DwArgs dw = {g->dZ1t, g->Xt, g->dZ2t, g->H1t, g->dOt, g->H2t, R, dw_rows(R), g->part, g->err};
  gemm_dw<<<dim3(DW_TILES, dw_splits(R)), DW_THREADS, DW_SMEM, st>>>(dw);
  if (lr > 0) g->step++;
  const FinishArgs f = {g->part, dw_splits(R), R, g->dZ1t, g->dZ2t, g->dOt, g->grad, g->master, g->adam_m, g->adam_v, g->packed,
                        lr, 1.f - powf(0.9f, (float)g->step), 1.f - powf(0.999f, (float)g->step)};
  dw_finish<<<FIN_BLOCKS, FIN_THREADS, 0, st>>>(f);
  CUDA_TRY(cudaGetLastError());
  if (grad_host) CUDA_TRY(cudaMemcpy(grad_host, g->grad, N_PARAMS * 4, cudaMemcpyDeviceToHost));
  float sums[4];  // waits for the step
  CUDA_TRY(cudaMemcpy(sums, g->acc, 16, cudaMemcpyDeviceToHost));
  int err = 0;
  memcpy(&err, sums + 3, 4);
  if (err) return fail(DDG_E_TIMEOUT, "guide: a tensor-core product did not complete (bounded wait)");
  if (stats3) memcpy(stats3, sums, 12);
  return DDG_OK;
}

int ddg_guide_predict(ddg_guide* g, const uint64_t* d_hands, int64_t n, int8_t* d_seed20, int8_t* d_hint20) {
  using namespace guide_nn;
  if (!g || (n > 0 && !d_hands)) return fail(DDG_E_ARG, "null argument");
  if (n < 0) return fail(DDG_E_ARG, "n < 0");
  CUDA_TRY(cudaSetDevice(g->device));
  int rc = guide_predict_on(g, d_hands, n, d_seed20, d_hint20, nullptr);
  if (rc) return rc;
  CUDA_TRY(cudaDeviceSynchronize());
  return check_err(g);
}

}  // extern "C"

// The inference of ddg_guide_predict on `stream`, waiting for that stream only: a guided
// stream calls it while its persistent solve kernel runs on another stream.
static int guide_predict_on(ddg_guide* g, const uint64_t* d_hands, int64_t n, int8_t* d_seed20, int8_t* d_hint20,
                            cudaStream_t stream) {
  using namespace guide_nn;
  CUDA_TRY(cudaMemsetAsync(g->err, 0, 4, stream));
  const int64_t total = n * 20;
  if (total > 0) {
    MlpArgs a;
    memset(&a, 0, sizeof(a));
    a.hands = d_hands;
    a.n = total;
    a.tiles = (int)tiles_of(total);
    a.packed = g->packed;
    a.master = g->master;
    a.seed20 = d_seed20;
    a.hint20 = d_hint20;
    a.err = g->err;
    mlp_rows<false><<<std::min(a.tiles, g->sms), MLP_THREADS<false>, MLP_SMEM, stream>>>(a);
    CUDA_TRY(cudaGetLastError());
  }
  if (stream) {
    CUDA_TRY(cudaStreamSynchronize(stream));
    return check_err(g);
  }
  return DDG_OK;
}

