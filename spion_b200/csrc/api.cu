// C ABI of spion_b200: contexts, the reference-layout entry points and the native ones.
// Orchestration only; kernels live in simt_fused.cu, mma_fused.cu, simt_attn.cu, structure.cu, pattern.cu, tc_fused.cu, tc_engine.cu.
//
// Pipelines (reference: Attention::attn_forward / attn_backward, models/block_attn.cu:453-545):
//   forward   S = Q K^T on the mask  ->  P = sparse row softmax(S)  ->  O = P V
//   backward  dP = dO V^T on the mask -> dS = softmax'(dP, P) -> dQ = dS K ; dK = dS^T Q ; dV = P^T dO
#include <atomic>
#include <mutex>
#include <new>
#include <unordered_map>
#include <vector>

#include "common.cuh"

namespace {
// The driver gives memory of a pool back to the system at the next synchronisation as soon as it has reserved more than the release
// threshold, and it counts what is in use: the threshold follows the memory in use, so that up to KEEP of free memory stays.
constexpr size_t KEEP = 64ull << 20;
struct DevicePool {
  cudaMemPool_t pool;
  cudaStream_t stream;
  std::mutex mutex;
  std::unordered_map<void*, size_t> sizes;        // what is in use
  size_t live = 0;
  std::vector<void*> waiting;                     // to be freed once the device can be waited for
  int follow() {
    uint64_t most = live + KEEP;
    return cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &most) == cudaSuccess ? SPION_OK : SPION_ERR_CUDA;
  }
};
// the pool of the current device, made on first use; nullptr if that failed
DevicePool* device_pool() {
  static std::mutex lock;
  static DevicePool* pools[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> hold(lock);
  if (!pools[dev]) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    DevicePool* d = new (std::nothrow) DevicePool();
    if (!d) return nullptr;
    if (cudaMemPoolCreate(&d->pool, &props) != cudaSuccess) { delete d; return nullptr; }
    if (d->follow() != SPION_OK || cudaStreamCreateWithFlags(&d->stream, cudaStreamNonBlocking) != cudaSuccess) {
      cudaMemPoolDestroy(d->pool);
      delete d;
      return nullptr;
    }
    pools[dev] = d;
  }
  return pools[dev];
}
}  // namespace

int device_alloc(void** p, size_t bytes) {
  *p = nullptr;
  DevicePool* d = device_pool();
  if (!d) return SPION_ERR_ALLOC;
  std::lock_guard<std::mutex> hold(d->mutex);
  if (cudaMallocFromPoolAsync(p, bytes, d->pool, d->stream) != cudaSuccess) { *p = nullptr; return SPION_ERR_ALLOC; }
  try {
    d->sizes.emplace(*p, bytes);
  } catch (...) {                                 // out of host memory: nothing may leave a C entry point
    cudaFreeAsync(*p, d->stream);
    *p = nullptr;
    return SPION_ERR_ALLOC;
  }
  d->live += bytes;
  d->follow();
  return cudaStreamSynchronize(d->stream) == cudaSuccess ? SPION_OK : SPION_ERR_ALLOC;   // usable on every stream from here on
}

void device_free(void* p) {
  if (!p) return;
  const bool idle = cudaDeviceSynchronize() == cudaSuccess;
  if (!idle) cudaGetLastError();                  // a stream of the device is being captured
  DevicePool* d = device_pool();
  if (!d) return;
  std::lock_guard<std::mutex> hold(d->mutex);
  try {
    d->waiting.push_back(p);
  } catch (...) { return; }
  if (!idle) return;                              // kernels may still use it: freed with the next one
  for (void* w : d->waiting) {
    const auto it = d->sizes.find(w);
    if (it != d->sizes.end()) { d->live -= it->second; d->sizes.erase(it); }
    cudaFreeAsync(w, d->stream);
  }
  d->waiting.clear();
  d->follow();
}

int scratch_alloc(void** p, size_t bytes, cudaStream_t st) {
  DevicePool* d = device_pool();
  if (d && cudaMallocFromPoolAsync(p, bytes, d->pool, st) == cudaSuccess) return SPION_OK;
  cudaGetLastError();
  *p = nullptr;
  return SPION_ERR_ALLOC;
}
void scratch_free(void* p, cudaStream_t st) { cudaFreeAsync(p, st); }

int sm_count() {
  static std::atomic<int> cached[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  int n = dev < 64 ? cached[dev].load() : 0;
  if (n) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (dev < 64) cached[dev].store(n);
  return n;
}

namespace {

struct DeviceGuard {
  int prev = -1;
  bool ok = true;
  explicit DeviceGuard(int dev) {
    if (cudaGetDevice(&prev) != cudaSuccess) { ok = false; return; }
    // Always, not only when the device differs: cudaSetDevice also binds the device's primary context to the
    // calling thread, which the driver entry point that encodes tensor maps needs (a thread of the autograd
    // engine that has not launched anything yet has no context bound, cudaGetDevice does not bind one).
    if (dev >= 0) ok = cudaSetDevice(dev) == cudaSuccess;
  }
  ~DeviceGuard() { if (prev >= 0) cudaSetDevice(prev); }
};

template <typename T>
bool dev_alloc(T** p, size_t n) { return device_alloc((void**)p, n * sizeof(T)) == SPION_OK; }

int rebuild_structure(spion_ctx* c) {
  c->launches += 1;
  return spion_launch_build_structure(c->mat, c->nb, c->nnzb_dev, c->row_ptr, c->col_idx, c->blk_row, c->col_ptr,
                                      c->row_idx, c->csc_pos, c->work, c->stream, c->nnzb_dev + 1);
}

bool is_dense(const spion_ctx* c) { return c->kind == SPION_KIND_DENSE || c->kind == SPION_KIND_DENSE_KPM; }
bool is_kpm(const spion_ctx* c) { return c->kind == SPION_KIND_DENSE_KPM || c->kind == SPION_KIND_BLOCK_KPM; }

}  // namespace

extern "C" const char* spion_status_string(int s) {
  switch (s) {
    case SPION_OK: return "ok";
    case SPION_ERR_ARG: return "bad argument";
    case SPION_ERR_SHAPE: return "unsupported shape";
    case SPION_ERR_CUDA: return "CUDA error";
    case SPION_ERR_TIMEOUT: return "device-side wait timed out";
    case SPION_ERR_UNSUPPORTED: return "combination not supported";
    case SPION_ERR_ALLOC: return "allocation failed";
    case SPION_ERR_STATE: return "call order";
    default: return "unknown status";
  }
}

extern "C" int spion_version(void) { return 100; }

extern "C" spion_ctx* spion_create(int kind, int head_dim, int seq_len, int num_batches, int block_size, int dtype,
                                   int device) {
  if (kind < SPION_KIND_DENSE || kind > SPION_KIND_BLOCK_KPM) return nullptr;
  if (head_dim < 1 || seq_len < 1 || num_batches < 1) return nullptr;
  if (dtype != SPION_F32 && dtype != SPION_BF16) return nullptr;
  const bool dense = kind == SPION_KIND_DENSE || kind == SPION_KIND_DENSE_KPM;
  int bs = block_size;
  if (dense) bs = (seq_len % 64 == 0) ? 64 : 32;          // internal tiling of the dense surface
  if (bs < 1 || seq_len % bs != 0) return nullptr;         // the reference truncates silently: int(L/bs)
  const int nb = seq_len / bs;
  if (nb > SPION_MAX_NB) return nullptr;

  DeviceGuard guard(device);
  if (!guard.ok) return nullptr;
  spion_ctx* c = new (std::nothrow) spion_ctx();
  if (!c) return nullptr;
  c->kind = kind; c->d = head_dim; c->L = seq_len; c->BH = num_batches; c->bs = bs; c->nb = nb;
  c->dtype = dtype; c->engine = SPION_ENGINE_AUTO;
  cudaGetDevice(&c->device);
  c->scale = 1.0f / sqrtf((float)head_dim);               // models/block_attn.cu:419
  c->stream = 0;
  c->nnzb = c->longest_col = -1;
  c->launches = 0;
  c->tc = nullptr;
  c->heads = 0;
  c->block32_path = 0;
  c->csr_stable = 0; c->csr_key[0] = c->csr_key[1] = c->csr_key[2] = nullptr; c->csr_nnz = -1;
  c->prof_on = 0; c->prof_n = 0;
  for (int i = 0; i < SPION_PROF_MAX_MARKS; ++i) { c->prof_ev[i] = nullptr; c->prof_stage[i] = -1; }
  for (int i = 0; i < SPION_STAGE_COUNT; ++i) { c->prof_ms[i] = 0; c->prof_cnt[i] = 0; }
  const size_t cap = (size_t)nb * nb;
  bool ok = dev_alloc(&c->mat, cap) && dev_alloc(&c->row_ptr, (size_t)nb + 1) && dev_alloc(&c->col_idx, cap) &&
            dev_alloc(&c->blk_row, cap) && dev_alloc(&c->col_ptr, (size_t)nb + 1) && dev_alloc(&c->row_idx, cap) &&
            dev_alloc(&c->csc_pos, cap) && dev_alloc(&c->work, cap) && dev_alloc(&c->nnzb_dev, 2) &&
            dev_alloc(&c->status_dev, 1);
  if (ok) ok = cudaMemset(c->status_dev, 0, sizeof(int)) == cudaSuccess;
  if (ok && dense) {
    ok = spion_launch_fill_mat(c->mat, (int)cap, 1, 0) == SPION_OK && rebuild_structure(c) == SPION_OK &&
         cudaStreamSynchronize(0) == cudaSuccess;
    c->nnzb = (int)cap;
  }
  if (!ok) { spion_destroy(c); return nullptr; }
  return c;
}

extern "C" void spion_destroy(spion_ctx* c) {
  if (!c) return;
  DeviceGuard guard(c->device);
  tc_engine_release(c);
  for (int i = 0; i < SPION_PROF_MAX_MARKS; ++i) if (c->prof_ev[i]) cudaEventDestroy(c->prof_ev[i]);
  device_free(c->mat); device_free(c->row_ptr); device_free(c->col_idx); device_free(c->blk_row); device_free(c->col_ptr);
  device_free(c->row_idx); device_free(c->csc_pos); device_free(c->work); device_free(c->nnzb_dev); device_free(c->status_dev);
  delete c;
}

extern "C" int spion_set_stream(spion_ctx* c, void* cuda_stream) {
  if (!c) return SPION_ERR_ARG;
  c->stream = (cudaStream_t)cuda_stream;
  return SPION_OK;
}

extern "C" int spion_set_engine(spion_ctx* c, int engine) {
  if (!c || engine < SPION_ENGINE_AUTO || engine > SPION_ENGINE_SIMT_STAGED) return SPION_ERR_ARG;
  if (engine == SPION_ENGINE_TCGEN05 && !tc_engine_supports(c)) return SPION_ERR_UNSUPPORTED;
  if ((engine == SPION_ENGINE_SIMT || engine == SPION_ENGINE_SIMT_STAGED) && c->heads != 0) return SPION_ERR_UNSUPPORTED;
  c->engine = engine;
  return SPION_OK;
}

extern "C" int spion_check_device_status(spion_ctx* c) {
  if (!c) return SPION_ERR_ARG;
  DeviceGuard guard(c->device);
  int word = 0;
  SPION_CUDA_TRY(cudaMemcpyAsync(&word, c->status_dev, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  SPION_CUDA_TRY(cudaStreamSynchronize(c->stream));
  const int linear = linear_status(1, c->stream);       // the layers around the attention share its stream
  if (word != 0) {
    SPION_CUDA_TRY(cudaMemsetAsync(c->status_dev, 0, sizeof(int), c->stream));
    fprintf(stderr, "spion_b200: device status word = 0x%x (a bounded wait gave up)\n", word);
    return SPION_ERR_TIMEOUT;
  }
  return linear;
}

extern "C" int spion_csr_arrays_are_stable(spion_ctx* c, int stable) {
  if (!c) return SPION_ERR_ARG;
  c->csr_stable = stable != 0;
  c->csr_key[0] = c->csr_key[1] = c->csr_key[2] = nullptr;
  c->csr_nnz = -1;
  return SPION_OK;
}

extern "C" int spion_set_head_layout(spion_ctx* c, int heads) {
  if (!c || heads < 0) return SPION_ERR_ARG;
  if (heads > 0) {
    if (is_dense(c) || !tc_engine_supports(c)) return SPION_ERR_UNSUPPORTED;   // the SIMT kernels address [BH, L, d] only
    if (c->BH % heads != 0) return SPION_ERR_SHAPE;
  }
  c->heads = heads;
  return SPION_OK;
}

extern "C" int spion_set_block32_path(spion_ctx* c, int path) {
  if (!c || path < 0 || path > 2) return SPION_ERR_ARG;
  c->block32_path = path;
  return SPION_OK;
}

extern "C" int spion_selftest_bounded_wait(spion_ctx* c, long long limit_cycles) {
  if (!c || limit_cycles < 1 || limit_cycles > 2000000000LL) return SPION_ERR_ARG;
  DeviceGuard guard(c->device);
  int rc = tc_engine_wait_selftest(c, limit_cycles);
  if (rc) return rc;
  return spion_check_device_status(c);      // expected: SPION_ERR_TIMEOUT, and the word is cleared again
}

extern "C" long long spion_launch_count(const spion_ctx* c) { return c ? c->launches : 0; }

// ------------------------------------------------------------ per-stage timing
int prof_drain(spion_ctx* c) {
  if (c->prof_n == 0) return SPION_OK;
  SPION_CUDA_TRY(cudaEventSynchronize(c->prof_ev[c->prof_n - 1]));
  for (int i = 1; i < c->prof_n; ++i) {
    const int st = c->prof_stage[i];
    if (st < 0) continue;
    float ms = 0.f;
    SPION_CUDA_TRY(cudaEventElapsedTime(&ms, c->prof_ev[i - 1], c->prof_ev[i]));
    c->prof_ms[st] += ms;
    c->prof_cnt[st] += 1;
  }
  c->prof_n = 0;
  return SPION_OK;
}

int prof_mark(spion_ctx* c, int stage) {
  if (!c->prof_on) return SPION_OK;
  if (stage < 0 && c->prof_n > SPION_PROF_MAX_MARKS - 16) {
    int rc = prof_drain(c);
    if (rc) return rc;
  }
  if (c->prof_n >= SPION_PROF_MAX_MARKS) return SPION_OK;
  if (!c->prof_ev[c->prof_n]) SPION_CUDA_TRY(cudaEventCreate(&c->prof_ev[c->prof_n]));
  SPION_CUDA_TRY(cudaEventRecord(c->prof_ev[c->prof_n], c->stream));
  c->prof_stage[c->prof_n] = stage;
  c->prof_n += 1;
  return SPION_OK;
}

extern "C" int spion_profile(spion_ctx* c, int enable) {
  if (!c) return SPION_ERR_ARG;
  DeviceGuard guard(c->device);
  if (!enable && c->prof_on) { int rc = prof_drain(c); if (rc) return rc; }
  c->prof_on = enable != 0;
  return SPION_OK;
}

extern "C" int spion_profile_get(spion_ctx* c, int stage, double* total_ms, long long* launches) {
  if (!c || stage < 0 || stage >= SPION_STAGE_COUNT) return SPION_ERR_ARG;
  DeviceGuard guard(c->device);
  int rc = prof_drain(c);
  if (rc) return rc;
  if (total_ms) *total_ms = c->prof_ms[stage];
  if (launches) *launches = c->prof_cnt[stage];
  return SPION_OK;
}

extern "C" int spion_profile_reset(spion_ctx* c) {
  if (!c) return SPION_ERR_ARG;
  DeviceGuard guard(c->device);
  int rc = prof_drain(c);
  for (int i = 0; i < SPION_STAGE_COUNT; ++i) { c->prof_ms[i] = 0; c->prof_cnt[i] = 0; }
  return rc;
}

extern "C" const char* spion_stage_name(int stage) {
  static const char* names[SPION_STAGE_COUNT] = {
      "structure", "sddmm_s", "softmax_fwd", "spmm_o", "sddmm_dp", "softmax_bwd", "spmm_dq", "spmm_dk", "spmm_dv",
      "fused_dp_ds", "spmm_dkdv", "fused_fwd", "bwd_row", "bwd_row_rc", "bwd_col_rc",
      "sddmm_softmax_fwd", "sddmm_softmax_bwd", "spmm_dqdkdv"};
  return (stage >= 0 && stage < SPION_STAGE_COUNT) ? names[stage] : "?";
}

// fp32 contexts run the fused SIMT kernels unless the per-stage ones are forced
static bool use_simt_fused(const spion_ctx* c, int value_mode) {
  return c->dtype == SPION_F32 && c->engine != SPION_ENGINE_SIMT_STAGED &&
         simt_fused_supports(c->bs, c->d, c->BH, value_mode);
}

// ============================================================ reference-layout sparse
// The block structure is derived from the caller's element CSR on every call: the reference's Python
// rebuilds those arrays for each forward (models/attention_blockcuda.py:26-43), usually into recycled
// allocations, so their addresses say nothing about their contents.  A caller that keeps the arrays
// alive and unchanged for as long as it passes them (spion_csr_arrays_are_stable) skips the rebuild
// when the same three pointers and nnz come back.
static int legacy_structure(spion_ctx* c, const int* offsets, const int* columns, const int* sum_mat, int nnz) {
  if (nnz < 0 || nnz % (c->bs * c->bs) != 0) return SPION_ERR_SHAPE;
  const int nnzb = nnz / (c->bs * c->bs);
  if (nnzb > c->nb * c->nb) return SPION_ERR_SHAPE;
  if (c->csr_stable && c->csr_key[0] == offsets && c->csr_key[1] == columns && c->csr_key[2] == sum_mat &&
      c->csr_nnz == nnz && c->nnzb == nnzb) {
    prof_mark(c, -1);
    return SPION_OK;
  }
  c->csr_key[0] = offsets; c->csr_key[1] = columns; c->csr_key[2] = sum_mat; c->csr_nnz = nnz;
  prof_mark(c, -1);
  int rc = spion_launch_mat_from_elemcsr(offsets, columns, sum_mat, c->nb, c->bs, c->mat, c->stream);
  if (rc) return rc;
  c->launches += 1;
  rc = rebuild_structure(c);
  if (rc) return rc;
  prof_mark(c, SPION_STAGE_STRUCTURE);
  c->nnzb = nnzb;
  c->longest_col = -1;
  return SPION_OK;
}

// The K operand of the forward and the V operand of the backward come transposed from the reference's Python, row-major from
// callers of the _rm forms.
static int block_forward(spion_ctx* c, const float* Q, const float* K, OperandLayout lk, const float* V, const float* keypad,
                         float* attn, float* out, const int* offsets, const int* columns, const int* sum_mat, int nnz) {
  if (!c || !Q || !K || !V || !attn || !out || !offsets || !columns || !sum_mat) return SPION_ERR_ARG;
  if (is_dense(c) || c->dtype != SPION_F32) return SPION_ERR_STATE;
  if (is_kpm(c) && !keypad) return SPION_ERR_ARG;
  DeviceGuard guard(c->device);
  int rc = legacy_structure(c, offsets, columns, sum_mat, nnz);
  if (rc) return rc;
  const Pattern p = ctx_pattern(c);
  const ValueLayout vl{VAL_ELEMCSR, c->L, (long long)nnz};
  const OperandLayout rm = row_major_operand(c->L, c->d);
  // floor of the running maximum: -100 (models/block_attn.cu:48) or 0 (models/block_attn_mask.cu:105)
  if (use_simt_fused(c, VAL_ELEMCSR)) {
    rc = simt_fused_forward(Q, rm, K, lk, V, rm, is_kpm(c) ? keypad : nullptr, is_kpm(c) ? 0.0f : -100.0f, attn, vl, out,
                            rm, p, c->BH, c->L, c->d, c->scale, c->stream, c->nnzb);
    if (!rc) prof_mark(c, SPION_STAGE_FUSED_FWD);
    c->launches += 1;
    return rc;
  }
  rc = simt_sddmm(SPION_F32, SPION_F32, Q, rm, K, lk, attn, vl, p, c->nnzb, c->BH, c->d, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SDDMM_S);
  if (rc) return rc;
  rc = softmax_fwd_rows(SPION_F32, attn, vl, attn, vl, p, c->BH, c->L, c->scale, is_kpm(c) ? keypad : nullptr,
                        is_kpm(c) ? 0.0f : -100.0f, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SOFTMAX_FWD);
  if (rc) return rc;
  rc = simt_spmm(SPION_F32, SPION_F32, false, attn, vl, V, rm, out, rm, p, c->BH, c->d, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SPMM_O);
  c->launches += 3;
  return rc;
}

static int block_backward(spion_ctx* c, const float* Q, const float* K, const float* V, OperandLayout lv, const float* P,
                          const float* O, const float* dO, float* dP_scratch, float* dS_scratch, float* dQ, float* dK,
                          float* dV, const int* offsets, const int* columns, const int* sum_mat, int nnz) {
  if (!c || !Q || !K || !V || !P || !dO || !dS_scratch || !dQ || !dK || !dV || !offsets || !columns || !sum_mat)
    return SPION_ERR_ARG;
  if (is_dense(c) || c->dtype != SPION_F32) return SPION_ERR_STATE;
  DeviceGuard guard(c->device);
  int rc = legacy_structure(c, offsets, columns, sum_mat, nnz);
  if (rc) return rc;
  const Pattern p = ctx_pattern(c);
  const ValueLayout vl{VAL_ELEMCSR, c->L, (long long)nnz};
  const OperandLayout rm = row_major_operand(c->L, c->d);
  if (use_simt_fused(c, VAL_ELEMCSR)) {
    c->launches += 2;
    return simt_fused_backward(Q, rm, K, rm, V, lv, P, vl, O, rm, dO, rm, dS_scratch, vl, dQ, rm, dK, rm, dV, rm, p, c->BH, c->d,
                               c->scale, c->stream, c, c->nnzb);
  }
  if (!dP_scratch) return SPION_ERR_ARG;
  rc = simt_sddmm(SPION_F32, SPION_F32, dO, rm, V, lv, dP_scratch, vl, p, c->nnzb, c->BH, c->d, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SDDMM_DP);
  if (rc) return rc;
  rc = softmax_bwd_rows(SPION_F32, dP_scratch, vl, P, vl, dS_scratch, vl, p, c->BH, c->L, c->scale, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SOFTMAX_BWD);
  if (rc) return rc;
  rc = simt_spmm(SPION_F32, SPION_F32, false, dS_scratch, vl, K, rm, dQ, rm, p, c->BH, c->d, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SPMM_DQ);
  if (rc) return rc;
  rc = simt_spmm(SPION_F32, SPION_F32, true, dS_scratch, vl, Q, rm, dK, rm, p, c->BH, c->d, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SPMM_DK);
  if (rc) return rc;
  rc = simt_spmm(SPION_F32, SPION_F32, true, P, vl, dO, rm, dV, rm, p, c->BH, c->d, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SPMM_DV);
  c->launches += 5;
  return rc;
}

extern "C" int spion_block_attn_forward(spion_ctx* c, const float* Q, const float* Kt, const float* V,
                                        const float* keypad, float* attn, float* out, const int* offsets,
                                        const int* columns, const int* sum_mat, int nnz) {
  if (!c) return SPION_ERR_ARG;
  return block_forward(c, Q, Kt, transposed_operand(c->L, c->d), V, keypad, attn, out, offsets, columns, sum_mat, nnz);
}

extern "C" int spion_block_attn_forward_rm(spion_ctx* c, const float* Q, const float* K, const float* V, const float* keypad,
                                           float* attn, float* out, const int* offsets, const int* columns,
                                           const int* sum_mat, int nnz) {
  if (!c) return SPION_ERR_ARG;
  return block_forward(c, Q, K, row_major_operand(c->L, c->d), V, keypad, attn, out, offsets, columns, sum_mat, nnz);
}

extern "C" int spion_block_attn_backward(spion_ctx* c, const float* Q, const float* K, const float* Vt, const float* P,
                                         const float* dO, float* dP_scratch, float* dS_scratch, float* dQ, float* dK,
                                         float* dV, const int* offsets, const int* columns, const int* sum_mat,
                                         int nnz) {
  if (!c || !dP_scratch) return SPION_ERR_ARG;
  return block_backward(c, Q, K, Vt, transposed_operand(c->L, c->d), P, nullptr, dO, dP_scratch, dS_scratch, dQ, dK, dV, offsets,
                        columns, sum_mat, nnz);
}

extern "C" int spion_block_attn_backward_rm(spion_ctx* c, const float* Q, const float* K, const float* V, const float* P,
                                            const float* O, const float* dO, float* dP_scratch, float* dS_scratch, float* dQ,
                                            float* dK, float* dV, const int* offsets, const int* columns, const int* sum_mat,
                                            int nnz) {
  if (!c) return SPION_ERR_ARG;
  return block_backward(c, Q, K, V, row_major_operand(c->L, c->d), P, O, dO, dP_scratch, dS_scratch, dQ, dK, dV, offsets, columns,
                        sum_mat, nnz);
}

extern "C" int spion_block_attn_needs_scratch(const spion_ctx* c) {
  return (c && !is_dense(c) && !use_simt_fused(c, VAL_ELEMCSR)) ? 1 : 0;
}

// ============================================================ reference-layout dense
static int dense_forward(spion_ctx* c, const float* Q, const float* K, const float* V, const float* keypad, float* attn,
                         float* out, OperandLayout lo) {
  if (!c || !Q || !K || !V || !attn || !out) return SPION_ERR_ARG;
  if (!is_dense(c) || c->dtype != SPION_F32) return SPION_ERR_STATE;
  if (is_kpm(c) && !keypad) return SPION_ERR_ARG;
  DeviceGuard guard(c->device);
  const Pattern p = ctx_pattern(c);
  const ValueLayout vl{VAL_DENSE_T, c->L, (long long)c->L * c->L};
  const OperandLayout rm = row_major_operand(c->L, c->d);
  const float* pad = is_kpm(c) ? keypad : nullptr;
  const bool joint = simt_dense_joint(false, c->L, c->d, c->BH, K, attn, attn);
  prof_mark(c, -1);
  // running-maximum floor -10 (models/attn.cu:21); key padding as models/attn_mask.cu:20
  int rc = joint ? simt_dense_scores(Q, lo, K, attn, c->BH, c->L, c->d, c->scale, pad, -10.0f, c->stream)
                 : simt_sddmm(SPION_F32, SPION_F32, Q, lo, K, rm, attn, vl, p, c->nnzb, c->BH, c->d, c->stream);
  if (rc) return rc;
  prof_mark(c, joint ? SPION_STAGE_S_SOFTMAX : SPION_STAGE_SDDMM_S);
  if (!joint) {
    rc = softmax_fwd_dense_t(attn, c->BH, c->L, c->scale, pad, -10.0f, c->stream);
    if (rc) return rc;
    prof_mark(c, SPION_STAGE_SOFTMAX_FWD);
  }
  rc = simt_spmm(SPION_F32, SPION_F32, false, attn, vl, V, lo, out, lo, p, c->BH, c->d, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SPMM_O);
  c->launches += joint ? 2 : 3;
  return rc;
}

static int dense_backward(spion_ctx* c, const float* Q, const float* K, const float* V, const float* attn, const float* dO,
                          float* s1, float* s3, float* dQ, float* dK, float* dV, OperandLayout lo) {
  if (!c || !Q || !K || !V || !attn || !dO || !s1 || !s3 || !dQ || !dK || !dV) return SPION_ERR_ARG;
  if (!is_dense(c) || c->dtype != SPION_F32) return SPION_ERR_STATE;
  DeviceGuard guard(c->device);
  const Pattern p = ctx_pattern(c);
  const ValueLayout vl{VAL_DENSE_T, c->L, (long long)c->L * c->L};
  const OperandLayout rm = row_major_operand(c->L, c->d);
  const bool joint = simt_dense_joint(true, c->L, c->d, c->BH, V, attn, s3);
  prof_mark(c, -1);
  int rc = joint ? simt_dense_dscores(dO, lo, V, attn, s3, c->BH, c->L, c->d, c->scale, c->stream)
                 : simt_sddmm(SPION_F32, SPION_F32, dO, lo, V, rm, s1, vl, p, c->nnzb, c->BH, c->d, c->stream);
  if (rc) return rc;
  prof_mark(c, joint ? SPION_STAGE_DP_SOFTMAX : SPION_STAGE_SDDMM_DP);
  if (!joint) {
    rc = softmax_bwd_dense_t(s1, attn, s3, c->BH, c->L, c->scale, c->stream);
    if (rc) return rc;
    prof_mark(c, SPION_STAGE_SOFTMAX_BWD);
  }
  c->launches += joint ? 1 : 2;
  rc = simt_dense_grads(attn, s3, Q, K, dO, lo, dQ, dK, dV, p, c->BH, c->L, c->d, c->stream);
  if (rc != SPION_ERR_UNSUPPORTED) {
    if (!rc) prof_mark(c, SPION_STAGE_DENSE_GRADS);
    c->launches += 1;
    return rc;
  }
  rc = simt_spmm(SPION_F32, SPION_F32, false, s3, vl, K, lo, dQ, lo, p, c->BH, c->d, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SPMM_DQ);
  if (rc) return rc;
  rc = simt_spmm(SPION_F32, SPION_F32, true, s3, vl, Q, lo, dK, lo, p, c->BH, c->d, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SPMM_DK);
  if (rc) return rc;
  rc = simt_spmm(SPION_F32, SPION_F32, true, attn, vl, dO, lo, dV, lo, p, c->BH, c->d, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SPMM_DV);
  c->launches += 3;
  return rc;
}

// The reference hands over Q, V, dO and takes the outputs as [BH, d, L] (K and, in the backward, V row-major; K transposed).
extern "C" int spion_dense_attn_forward(spion_ctx* c, const float* Qt, const float* K, const float* Vt,
                                        const float* keypad, float* attn, float* out) {
  if (!c) return SPION_ERR_ARG;
  return dense_forward(c, Qt, K, Vt, keypad, attn, out, transposed_operand(c->L, c->d));
}

extern "C" int spion_dense_attn_backward(spion_ctx* c, const float* Qt, const float* Kt, const float* V,
                                         const float* attn, const float* dOt, float* s1, float* s2, float* s3,
                                         float* dQt, float* dKt, float* dVt) {
  (void)s2;
  if (!c) return SPION_ERR_ARG;
  return dense_backward(c, Qt, Kt, V, attn, dOt, s1, s3, dQt, dKt, dVt, transposed_operand(c->L, c->d));
}

extern "C" int spion_dense_attn_forward_rm(spion_ctx* c, const float* Q, const float* K, const float* V, const float* keypad,
                                           float* attn, float* out) {
  if (!c) return SPION_ERR_ARG;
  return dense_forward(c, Q, K, V, keypad, attn, out, row_major_operand(c->L, c->d));
}

extern "C" int spion_dense_attn_backward_rm(spion_ctx* c, const float* Q, const float* K, const float* V, const float* attn,
                                            const float* O, const float* dO, float* s1, float* s3, float* dQ, float* dK,
                                            float* dV) {
  (void)O;
  if (!c) return SPION_ERR_ARG;
  return dense_backward(c, Q, K, V, attn, dO, s1, s3, dQ, dK, dV, row_major_operand(c->L, c->d));
}

extern "C" long long spion_dense_attn_scratch_floats(const spion_ctx* c) { return c ? (long long)c->BH * c->L * c->L : 0; }

__global__ void k_expand_keypad(const float* __restrict__ mask, int heads, int L, long long n, float* __restrict__ pen) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long bh = i / L;
    pen[i] = 1e6f * (1.0f - mask[(bh / heads) * L + (i - bh * L)]);
  }
}

extern "C" int spion_expand_keypad(const float* mask, int batch, int heads, int L, float* pen, void* cuda_stream) {
  if (!mask || !pen || batch < 1 || heads < 1 || L < 1) return SPION_ERR_ARG;
  const long long n = (long long)batch * heads * L;
  const long long blocks = (n + 255) / 256;
  k_expand_keypad<<<(unsigned)(blocks < 1184 ? blocks : 1184), 256, 0, (cudaStream_t)cuda_stream>>>(mask, heads, L, n, pen);
  SPION_LAUNCH_CHECK();
  return SPION_OK;
}

// ============================================================ native (block-tile) API
extern "C" int spion_set_pattern(spion_ctx* c, const uint8_t* mat) {
  if (!c || !mat) return SPION_ERR_ARG;
  if (is_dense(c)) return SPION_ERR_STATE;
  DeviceGuard guard(c->device);
  SPION_CUDA_TRY(cudaMemcpyAsync(c->mat, mat, (size_t)c->nb * c->nb, cudaMemcpyDeviceToDevice, c->stream));
  int rc = rebuild_structure(c);
  if (rc) return rc;
  int32_t n[2] = {0, 0};
  SPION_CUDA_TRY(cudaMemcpyAsync(n, c->nnzb_dev, sizeof(n), cudaMemcpyDeviceToHost, c->stream));
  SPION_CUDA_TRY(cudaStreamSynchronize(c->stream));
  c->nnzb = n[0];
  c->longest_col = n[1];
  if (tc_engine_supports(c)) {
    rc = tc_engine_prepare(c);
    if (rc) return rc;
  }
  return SPION_OK;
}

extern "C" int spion_pattern_nnzb(const spion_ctx* c) { return c ? c->nnzb : SPION_ERR_ARG; }

static bool use_tc(const spion_ctx* c) {
  if (c->engine == SPION_ENGINE_SIMT || c->engine == SPION_ENGINE_SIMT_STAGED) return false;
  return tc_engine_supports(c);
}

extern "C" int spion_attn_forward_ex(spion_ctx* c, const void* Q, const void* K, const void* V, const float* keypad,
                                     void* P, void* O, float* S_scratch) {
  if (!c || !Q || !K || !V || !P || !O) return SPION_ERR_ARG;
  if (is_dense(c) || c->nnzb < 0) return SPION_ERR_STATE;
  DeviceGuard guard(c->device);
  if (use_tc(c)) return tc_engine_forward(c, Q, K, V, keypad, P, O, S_scratch);
  if (c->heads != 0) return SPION_ERR_UNSUPPORTED;
  const Pattern p = ctx_pattern(c);
  const long long nnz = (long long)c->nnzb * c->bs * c->bs;
  const ValueLayout vl{VAL_BLOCKTILE, c->L, nnz};
  const OperandLayout rm = row_major_operand(c->L, c->d);
  prof_mark(c, -1);
  if (use_simt_fused(c, VAL_BLOCKTILE)) {
    int rc = simt_fused_forward((const float*)Q, rm, (const float*)K, rm, (const float*)V, rm, keypad,
                                keypad ? 0.0f : -100.0f, (float*)P, vl, (float*)O, rm, p, c->BH, c->L, c->d, c->scale,
                                c->stream, c->nnzb);
    if (!rc) prof_mark(c, SPION_STAGE_FUSED_FWD);
    c->launches += 1;
    return rc;
  }
  if (!S_scratch) return SPION_ERR_ARG;
  int rc = simt_sddmm(c->dtype, SPION_F32, Q, rm, K, rm, S_scratch, vl, p, c->nnzb, c->BH, c->d, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SDDMM_S);
  if (rc) return rc;
  rc = softmax_fwd_rows(c->dtype, S_scratch, vl, P, vl, p, c->BH, c->L, c->scale, keypad, keypad ? 0.0f : -100.0f,
                        c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SOFTMAX_FWD);
  if (rc) return rc;
  rc = simt_spmm(c->dtype, c->dtype, false, P, vl, V, rm, O, rm, p, c->BH, c->d, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SPMM_O);
  c->launches += 3;
  return rc;
}

extern "C" int spion_attn_backward_ex(spion_ctx* c, const void* Q, const void* K, const void* V, const void* P,
                                      const void* O, const void* dO, void* dS, float* dP_scratch, float* delta,
                                      void* dQ, void* dK, void* dV) {
  if (!c || !Q || !K || !V || !P || !dO || !dS || !dQ || !dK || !dV) return SPION_ERR_ARG;
  if (is_dense(c) || c->nnzb < 0) return SPION_ERR_STATE;
  DeviceGuard guard(c->device);
  if (use_tc(c)) {
    if (!O) return SPION_ERR_ARG;
    (void)delta;
    return tc_engine_backward(c, Q, K, V, P, O, dO, dS, dP_scratch, dQ, dK, dV);
  }
  if (c->heads != 0) return SPION_ERR_UNSUPPORTED;
  const Pattern p = ctx_pattern(c);
  const long long nnz = (long long)c->nnzb * c->bs * c->bs;
  const ValueLayout vl{VAL_BLOCKTILE, c->L, nnz};
  const OperandLayout rm = row_major_operand(c->L, c->d);
  prof_mark(c, -1);
  if (use_simt_fused(c, VAL_BLOCKTILE)) {
    c->launches += 2;
    return simt_fused_backward((const float*)Q, rm, (const float*)K, rm, (const float*)V, rm, (const float*)P, vl,
                               (const float*)O, rm, (const float*)dO, rm, (float*)dS, vl, (float*)dQ, rm, (float*)dK, rm, (float*)dV, rm, p,
                               c->BH, c->d, c->scale, c->stream, c, c->nnzb);
  }
  if (!dP_scratch) return SPION_ERR_ARG;
  int rc = simt_sddmm(c->dtype, SPION_F32, dO, rm, V, rm, dP_scratch, vl, p, c->nnzb, c->BH, c->d, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SDDMM_DP);
  if (rc) return rc;
  rc = softmax_bwd_rows(c->dtype, dP_scratch, vl, P, vl, dS, vl, p, c->BH, c->L, c->scale, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SOFTMAX_BWD);
  if (rc) return rc;
  rc = simt_spmm(c->dtype, c->dtype, false, dS, vl, K, rm, dQ, rm, p, c->BH, c->d, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SPMM_DQ);
  if (rc) return rc;
  rc = simt_spmm(c->dtype, c->dtype, true, dS, vl, Q, rm, dK, rm, p, c->BH, c->d, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SPMM_DK);
  if (rc) return rc;
  rc = simt_spmm(c->dtype, c->dtype, true, P, vl, dO, rm, dV, rm, p, c->BH, c->d, c->stream);
  if (!rc) prof_mark(c, SPION_STAGE_SPMM_DV);
  c->launches += 5;
  return rc;
}

extern "C" int spion_needs_scratch(const spion_ctx* c) {
  if (!c || is_dense(c)) return 0;
  return (use_tc(c) || use_simt_fused(c, VAL_BLOCKTILE)) ? 0 : 1;
}

extern "C" int spion_supports_fused(const spion_ctx* c) {
  return (c && !is_dense(c) && use_tc(c)) ? 1 : 0;
}

extern "C" int spion_attn_forward_fused(spion_ctx* c, const void* Q, const void* K, const void* V, const float* keypad,
                                        void* O, float* lse, void* P_optional) {
  if (!c || !Q || !K || !V || !O || !lse) return SPION_ERR_ARG;
  if (is_dense(c) || c->nnzb < 0) return SPION_ERR_STATE;
  if (!use_tc(c)) return SPION_ERR_UNSUPPORTED;
  DeviceGuard guard(c->device);
  return tc_engine_forward_fused(c, Q, K, V, keypad, O, lse, P_optional);
}

extern "C" int spion_attn_backward_fused(spion_ctx* c, const void* Q, const void* K, const void* V, const void* O,
                                         const void* dO, const float* lse, const float* keypad, void* dQ, void* dK,
                                         void* dV) {
  if (!c || !Q || !K || !V || !O || !dO || !lse || !dQ || !dK || !dV) return SPION_ERR_ARG;
  if (is_dense(c) || c->nnzb < 0) return SPION_ERR_STATE;
  if (!use_tc(c)) return SPION_ERR_UNSUPPORTED;
  DeviceGuard guard(c->device);
  return tc_engine_backward_fused(c, Q, K, V, O, dO, lse, keypad, dQ, dK, dV);
}

extern "C" int spion_attn_forward_probs(spion_ctx* c, const void* Q, const void* K, const void* V, const float* keypad, void* O, float* lse,
                                        void* P_optional, float* stat) {
  if (!c || !Q || !K || !V || !O || !stat) return SPION_ERR_ARG;
  if (is_dense(c) || c->nnzb < 0) return SPION_ERR_STATE;
  if (!use_tc(c)) return SPION_ERR_UNSUPPORTED;
  DeviceGuard guard(c->device);
  return tc_engine_forward_probs(c, Q, K, V, keypad, O, lse, P_optional, stat);
}

extern "C" int spion_attn_backward_probs(spion_ctx* c, const void* Q, const void* K, const void* V, const void* O, const void* dO, const float* stat,
                                         const float* keypad, void* dQ, void* dK, void* dV) {
  if (!c || !Q || !K || !V || !O || !dO || !stat || !dQ || !dK || !dV) return SPION_ERR_ARG;
  if (is_dense(c) || c->nnzb < 0) return SPION_ERR_STATE;
  if (!use_tc(c)) return SPION_ERR_UNSUPPORTED;
  DeviceGuard guard(c->device);
  return tc_engine_backward_probs(c, Q, K, V, O, dO, stat, keypad, dQ, dK, dV);
}

extern "C" int spion_block32_path_in_use(const spion_ctx* c) {
  if (!c) return SPION_ERR_ARG;
  return use_tc(c) ? tc_engine_block32_path(c) : 0;
}

extern "C" int spion_mean_map_recompute(spion_ctx* c, const void* Q, const void* K, const float* lse,
                                        const float* keypad, float* A) {
  if (!c || !Q || !K || !lse || !A) return SPION_ERR_ARG;
  if (is_dense(c) || c->nnzb < 0) return SPION_ERR_STATE;
  if (!use_tc(c)) return SPION_ERR_UNSUPPORTED;
  DeviceGuard guard(c->device);
  return tc_engine_mean_map(c, Q, K, lse, keypad, A);
}

extern "C" int spion_softmax_forward_ex(spion_ctx* c, const float* S, const float* keypad, void* P) {
  if (!c || !S || !P) return SPION_ERR_ARG;
  if (is_dense(c) || c->nnzb < 0) return SPION_ERR_STATE;
  DeviceGuard guard(c->device);
  const ValueLayout vl{VAL_BLOCKTILE, c->L, (long long)c->nnzb * c->bs * c->bs};
  c->launches += 1;
  return softmax_fwd_rows(c->dtype, S, vl, P, vl, ctx_pattern(c), c->BH, c->L, c->scale, keypad,
                          keypad ? 0.0f : -100.0f, c->stream);
}

extern "C" int spion_softmax_backward_ex(spion_ctx* c, const float* dP, const void* P, void* dS) {
  if (!c || !dP || !P || !dS) return SPION_ERR_ARG;
  if (is_dense(c) || c->nnzb < 0) return SPION_ERR_STATE;
  DeviceGuard guard(c->device);
  const ValueLayout vl{VAL_BLOCKTILE, c->L, (long long)c->nnzb * c->bs * c->bs};
  c->launches += 1;
  return softmax_bwd_rows(c->dtype, dP, vl, P, vl, dS, vl, ctx_pattern(c), c->BH, c->L, c->scale, c->stream);
}
