// leco_batch.cu -- batch engine: thousands of columns of uneven length, mixed
// uint32/uint64 and mixed LeCo/FOR/Delta/poly codecs, encoded and decoded by
// one persistent launch per pass.
//
// Work queue: the batch's blocks are listed column by column as work items.  A decoder
// item is 256/G consecutive blocks, G being the column's threads per block (32, 64, 128
// or 256): one block per item for G = 256, eight for G = 32 (one warp each).  An encoder
// item is 256/R consecutive blocks of R rows of 32 values (leco_rows.cuh: one thread per
// row), or one block of 512 rows in a launch of its own.  Every CTA of a persistent grid
// takes the next item from an atomic ticket and runs the encoder or decoder instance for
// that column's codec and value type (decoder: G and unroll depth too).  Items are handed
// out in order and every CTA of the grid is resident, so the encoder's per-column
// look-back (byte offsets, one word per item) only ever waits on items that are already
// being processed.  The reference's sequential fits are part of the encoder item
// (rows_fit): as a pass of their own, one lane per block, they took 606 of the 949 us of an
// encode + decode pass over 20 columns of 64K-4M values; the whole pass takes 162 us now.
// Every CTA of an encode launch has the shared memory of the batch's largest item: three CTAs
// per SM with LeCo, FOR and Delta columns, two for all of them when one is u64 degree-2 in large
// blocks.  The encode kernel holds every codec's encoder in 80 registers and spills some of them.
//
// The reference has no counterpart: its drivers loop over blocks of one column
// (experiments/leco_int_fix_template.cpp:111-127, :145-153).  The per-column
// path (leco_batch_*_per_column) is what a caller of leco_encode / leco_decode
// does without the batch engine, kept as the baseline.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <vector>

#include "leco_batch.cuh"

using namespace leco;

struct leco_batch {
  std::vector<leco_column_desc> cols;
  std::vector<uint64_t> prefix;
  int fit_mode = LECO_FIT_REFERENCE;
  int device = 0;
  DevCol *d_cols = nullptr;
  uint64_t *d_prefix = nullptr;
  uint64_t *d_items = nullptr, *d_enc_items = nullptr;
  uint64_t nitems = 0, enc_n[2] = {0, 0};
  uint8_t *d_ws = nullptr;  // status [encoder items] | tickets
  uint64_t ws_bytes = 0, status_bytes = 0;
  uint32_t enc_smem[2] = {0, 0};
  int enc_grid[2] = {0, 0}, dec_grid = 0;
  uint32_t *err = nullptr;               // library error word on this device
  cudaStream_t capture_stream = nullptr;  // graphs are captured here (the caller's stream may be the legacy default stream)
  cudaGraphExec_t graph[4] = {nullptr, nullptr, nullptr, nullptr};
};

namespace {

// What a column's (block size, group_threads) may ask for: see the rule in leco_batch_create.
constexpr uint32_t kBatchMaxSmem = 200 * 1024;

// The most shared memory an encoder item can take (any codec, value type and block size).  A
// kernel's opt-in to more than 48 KB belongs to the kernel, not to the batch: set to one batch's
// own size it would take a smaller batch's after that one was made.
int batch_enc_max_smem(int which) {
  uint32_t m = 0;
  for (uint32_t R = which ? 512 : 8; R <= (which ? 512u : 256u); R <<= 1) m = std::max(m, rows_layout(which ? 512 : 256, R, 8, 3).total);
  return (int)m;
}

int berr(int code, const std::string &m) { return leco::record_error(code, m); }

bool needs_seq(int codec, int dtype, uint32_t bs, int fit_mode) {
  if (fit_mode != LECO_FIT_REFERENCE) return false;
  if (codec == kLinear) return !(dtype == LECO_U32 && bs <= 2048);
  return codec == kPoly2;
}

BatchArgs args_of(const leco_batch *b, uint32_t *err) {
  BatchArgs B;
  B.cols = b->d_cols;
  B.prefix = b->d_prefix;
  B.items = b->d_items;
  B.enc_items = b->d_enc_items;
  B.enc_n[0] = b->enc_n[0];
  B.enc_n[1] = b->enc_n[1];
  B.nitems = b->nitems;
  B.ncols = (uint32_t)b->cols.size();
  B.total = b->prefix.back();
  B.status = reinterpret_cast<uint64_t *>(b->d_ws);
  B.ticket = reinterpret_cast<unsigned long long *>(b->d_ws + b->status_bytes);
  B.error = err;
  return B;
}

}  // namespace

extern "C" {

int leco_batch_create(const leco_column_desc *h_cols, uint32_t ncols, int fit_mode, leco_batch **out) {
  if (!h_cols || !ncols || !out) return berr(LECO_ERR_ARG, "leco_batch_create: null pointer or empty batch");
  if (fit_mode != LECO_FIT_REFERENCE && fit_mode != LECO_FIT_EXACT) return berr(LECO_ERR_ARG, "leco_batch_create: bad fit_mode");
  auto *b = new leco_batch();
  b->cols.assign(h_cols, h_cols + ncols);
  b->fit_mode = fit_mode;
  cudaGetDevice(&b->device);
  b->prefix.resize(ncols + 1);
  std::vector<DevCol> dc(ncols);
  uint64_t total = 0;
  for (uint32_t i = 0; i < ncols; ++i) {
    const leco_column_desc &c = h_cols[i];
    if (c.codec < kLinear || c.codec > kPoly2 || (c.dtype != 4 && c.dtype != 8) || !c.block_size ||
        c.block_size > LECO_MAX_BLOCK || !c.n || !c.d_payload || !c.d_offsets) {
      delete b;
      return berr(LECO_ERR_ARG, "leco_batch_create: bad descriptor for column " + std::to_string(i));
    }
    b->prefix[i] = total;
    total += leco_num_blocks(c.n, c.block_size);
    DevCol &d = dc[i];
    d.codec = c.codec;
    d.dtype = c.dtype;
    d.bs = c.block_size;
    d.seq = needs_seq(c.codec, c.dtype, c.block_size, fit_mode);
    d.n = c.n;
    d.values = c.d_values;
    d.out = c.d_out;
    d.payload = c.d_payload;
    d.payload_cap = c.payload_cap;
    d.offsets = c.d_offsets;
    d.dir = c.d_dir;
    for (int k = 0; k < 10; ++k) d.polyX[k] = 0;
    if (c.codec == kPoly2) {
      const uint64_t nb = leco_num_blocks(c.n, c.block_size);
      poly2_x_sums((uint32_t)std::min<uint64_t>(c.n, c.block_size), d.polyX);
      poly2_x_sums((uint32_t)(c.n - (nb - 1) * c.block_size), d.polyX + 5);
    }
    d.group = c.group_threads ? c.group_threads : (c.block_size <= kWarpBlock ? 32u : 256u);
    d.unroll = c.unroll ? c.unroll : 2u;
    d.rows = rows_threads(c.block_size);
    d.pad = 0;
    if ((d.group != 32 && d.group != 64 && d.group != 128 && d.group != 256) ||
        (d.unroll != 1 && d.unroll != 2 && d.unroll != 4)) {
      delete b;
      return berr(LECO_ERR_ARG, "leco_batch_create: column " + std::to_string(i) +
                                    ": group_threads must be 0, 32, 64, 128 or 256 and unroll 0, 1, 2 or 4");
    }
    // The rule for group_threads of the interface: its blocks' values, one slice for each group of
    // a 256-thread CTA, within 200 KB.  (Neither kernel lays its items out so: the encoder's follow
    // the block size alone, the decoder's need no shared memory.)
    const uint32_t slice = (enc_smem_bytes(c.block_size, (uint32_t)c.dtype) + 15) / 16 * 16;
    const uint32_t item_smem = slice * (256 / d.group);
    if (item_smem > kBatchMaxSmem) {
      delete b;
      return berr(LECO_ERR_ARG, "leco_batch_create: column " + std::to_string(i) + ": " + std::to_string(256 / d.group) +
                                    " groups of " + std::to_string(slice) + " bytes of shared memory exceed the " +
                                    std::to_string(kBatchMaxSmem) + " a CTA may use");
    }
    const int which = d.rows == 512;
    b->enc_smem[which] = std::max(b->enc_smem[which], rows_layout(which ? 512 : 256, d.rows, (uint32_t)c.dtype,
                                                                  (uint32_t)rows_sums(c.codec)).total);
  }
  // work items: (column << 32) | first block, 256/G blocks per item
  std::vector<uint64_t> items;
  for (uint32_t i = 0; i < ncols; ++i) {
    const uint64_t nb = leco_num_blocks(h_cols[i].n, h_cols[i].block_size);
    const uint64_t step = 256 / dc[i].group;
    for (uint64_t blk = 0; blk < nb; blk += step) items.push_back(((uint64_t)i << 32) | blk);
  }
  // encoder items: (column << 32) | item, items of 256 threads before those of 512
  std::vector<uint64_t> enc_items;
  for (int which = 0; which < 2; ++which) {
    for (uint32_t i = 0; i < ncols; ++i) {
      if ((dc[i].rows == 512) != (which == 1)) continue;
      const uint64_t nb = leco_num_blocks(h_cols[i].n, h_cols[i].block_size), per = which ? 1 : 256 / dc[i].rows;
      dc[i].item0 = enc_items.size();
      for (uint64_t k = 0; k * per < nb; ++k) enc_items.push_back(((uint64_t)i << 32) | k);
    }
    b->enc_n[which] = enc_items.size() - (which ? b->enc_n[0] : 0);
  }
  b->nitems = items.size();
  b->prefix[ncols] = total;
  if (total > 0xffffffffull) {
    delete b;
    return berr(LECO_ERR_ARG, "leco_batch_create: more than 2^32 blocks");
  }
  b->status_bytes = (enc_items.size() * 8 + 255) / 256 * 256;
  b->ws_bytes = b->status_bytes + 256;
  // the per-column calls encode through the same workspace
  for (uint32_t i = 0; i < ncols; ++i)
    b->ws_bytes = std::max(b->ws_bytes, leco_encode_workspace_bytes(h_cols[i].codec, h_cols[i].dtype, h_cols[i].n,
                                                                    h_cols[i].block_size, fit_mode));
  cudaError_t e = cudaMalloc(&b->d_cols, ncols * sizeof(DevCol));
  if (e == cudaSuccess) e = cudaMalloc(&b->d_prefix, (ncols + 1) * sizeof(uint64_t));
  if (e == cudaSuccess) e = cudaMalloc(&b->d_ws, b->ws_bytes);
  if (e == cudaSuccess) e = cudaMemcpy(b->d_cols, dc.data(), ncols * sizeof(DevCol), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b->d_prefix, b->prefix.data(), (ncols + 1) * sizeof(uint64_t), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMalloc(&b->d_items, std::max<size_t>(1, items.size()) * sizeof(uint64_t));
  if (e == cudaSuccess) e = cudaMemcpy(b->d_items, items.data(), items.size() * sizeof(uint64_t), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMalloc(&b->d_enc_items, std::max<size_t>(1, enc_items.size()) * sizeof(uint64_t));
  if (e == cudaSuccess)
    e = cudaMemcpy(b->d_enc_items, enc_items.data(), enc_items.size() * sizeof(uint64_t), cudaMemcpyHostToDevice);
  if (e == cudaSuccess && leco::device_error_word(&b->err)) e = cudaErrorUnknown;
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&b->capture_stream, cudaStreamNonBlocking);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(batch_encode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, batch_enc_max_smem(0));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(batch_encode_large_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, batch_enc_max_smem(1));
  int sms = 148, per_enc[2] = {1, 1}, per_dec = 1;
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->device);
  if (e == cudaSuccess && b->enc_n[0])
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_enc[0], batch_encode_kernel, 256, b->enc_smem[0]);
  if (e == cudaSuccess && b->enc_n[1])
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_enc[1], batch_encode_large_kernel, 512, b->enc_smem[1]);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_dec, batch_decode_kernel, 256, 0);
  if (e != cudaSuccess || per_enc[0] < 1 || per_enc[1] < 1 || per_dec < 1) {
    leco_batch_destroy(b);
    return berr(e != cudaSuccess ? LECO_ERR_CUDA : LECO_ERR_ARG,
                std::string("leco_batch_create: ") + (e != cudaSuccess ? cudaGetErrorString(e) : "no resident CTA fits"));
  }
  // every CTA of the persistent grid must be resident (the look-back waits on them)
  for (int which = 0; which < 2; ++which)
    b->enc_grid[which] = (int)std::min<uint64_t>(b->enc_n[which], (uint64_t)sms * per_enc[which]);
  b->dec_grid = (int)std::min<uint64_t>(b->nitems, (uint64_t)sms * per_dec);
  *out = b;
  return LECO_OK;
}

int leco_batch_destroy(leco_batch *b) {
  if (!b) return LECO_OK;
  for (auto &g : b->graph)
    if (g) cudaGraphExecDestroy(g);
  if (b->capture_stream) cudaStreamDestroy(b->capture_stream);
  if (b->d_cols) cudaFree(b->d_cols);
  if (b->d_prefix) cudaFree(b->d_prefix);
  if (b->d_items) cudaFree(b->d_items);
  if (b->d_enc_items) cudaFree(b->d_enc_items);
  if (b->d_ws) cudaFree(b->d_ws);
  delete b;
  return LECO_OK;
}

uint64_t leco_batch_total_blocks(const leco_batch *b) { return b ? b->prefix.back() : 0; }

int leco_batch_encode(leco_batch *b, leco_stream_t stream) {
  if (!b) return berr(LECO_ERR_ARG, "leco_batch_encode: null batch");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const BatchArgs B = args_of(b, b->err);
  cudaError_t e = cudaMemsetAsync(b->d_ws, 0, b->status_bytes + 256, st);  // look-back words + ticket
  if (e == cudaSuccess && b->enc_grid[0]) batch_encode_kernel<<<b->enc_grid[0], 256, b->enc_smem[0], st>>>(B);
  if (e == cudaSuccess && b->enc_grid[1]) batch_encode_large_kernel<<<b->enc_grid[1], 512, b->enc_smem[1], st>>>(B);
  if (e == cudaSuccess) e = cudaGetLastError();
  return e == cudaSuccess ? LECO_OK : berr(LECO_ERR_CUDA, std::string("leco_batch_encode: ") + cudaGetErrorString(e));
}

int leco_batch_decode(leco_batch *b, leco_stream_t stream) {
  if (!b) return berr(LECO_ERR_ARG, "leco_batch_decode: null batch");
  for (const auto &c : b->cols) {
    if (!c.d_out) return berr(LECO_ERR_ARG, "leco_batch_decode: a column has no output buffer");
    if (reinterpret_cast<uintptr_t>(c.d_out) & (uint64_t)(c.dtype - 1))  // values are stored as 16/32-byte vectors
      return berr(LECO_ERR_ARG, "leco_batch_decode: a column's output buffer is not aligned to its value size");
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const BatchArgs B = args_of(b, b->err);
  cudaError_t e = cudaMemsetAsync(b->d_ws + b->status_bytes, 0, 256, st);  // ticket
  if (e == cudaSuccess) batch_decode_kernel<<<b->dec_grid, 256, 0, st>>>(B);
  if (e == cudaSuccess) e = cudaGetLastError();
  return e == cudaSuccess ? LECO_OK : berr(LECO_ERR_CUDA, std::string("leco_batch_decode: ") + cudaGetErrorString(e));
}

int leco_batch_run_graph(leco_batch *b, int passes, leco_stream_t stream) {
  if (!b || passes < 1 || passes > 3) return berr(LECO_ERR_ARG, "leco_batch_run_graph: passes must be 1 (encode), 2 (decode) or 3");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (!b->graph[passes]) {
    cudaGraph_t g = nullptr;
    cudaStream_t cs = b->capture_stream;
    leco_stream_t lcs = reinterpret_cast<leco_stream_t>(cs);
    cudaError_t e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return berr(LECO_ERR_CUDA, std::string("leco_batch_run_graph: ") + cudaGetErrorString(e));
    int rc = LECO_OK;
    if (passes & 1) rc = leco_batch_encode(b, lcs);
    if (!rc && (passes & 2)) rc = leco_batch_decode(b, lcs);
    e = cudaStreamEndCapture(cs, &g);
    if (rc) {
      if (g) cudaGraphDestroy(g);
      return rc;
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&b->graph[passes], g, 0);
    if (g) cudaGraphDestroy(g);
    if (e != cudaSuccess) return berr(LECO_ERR_CUDA, std::string("leco_batch_run_graph: ") + cudaGetErrorString(e));
  }
  cudaError_t e = cudaGraphLaunch(b->graph[passes], st);
  return e == cudaSuccess ? LECO_OK : berr(LECO_ERR_CUDA, std::string("leco_batch_run_graph: ") + cudaGetErrorString(e));
}

// Baseline: one leco_encode call per column (the batch's workspace is reused;
// each call resets it).
int leco_batch_encode_per_column(leco_batch *b, leco_stream_t stream) {
  if (!b) return berr(LECO_ERR_ARG, "null batch");
  for (const auto &c : b->cols) {
    int rc = leco_encode(c.codec, c.dtype, c.d_values, c.n, c.block_size, b->fit_mode, c.d_payload, c.payload_cap,
                         c.d_offsets, c.d_dir, b->d_ws, b->ws_bytes, stream);
    if (rc) return rc;
  }
  return LECO_OK;
}

int leco_batch_decode_per_column(leco_batch *b, leco_stream_t stream) {
  if (!b) return berr(LECO_ERR_ARG, "null batch");
  for (const auto &c : b->cols) {
    int rc = leco_decode(c.codec, c.dtype, c.d_payload, c.d_offsets, c.n, c.block_size, c.d_out, stream);
    if (rc) return rc;
  }
  return LECO_OK;
}

}  // extern "C"
