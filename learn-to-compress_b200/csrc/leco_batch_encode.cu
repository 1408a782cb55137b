// leco_batch_encode.cu -- the batch engine's persistent encode kernel (see
// leco_batch.cu for the work queue).  A translation unit of its own: its per-codec
// encoder instances compile in parallel with the decoder's.
#include "leco_batch.cuh"

namespace leco {

template <typename T, int CODEC>
__device__ __forceinline__ void batch_encode_one(const BatchArgs &B, const DevCol &c, uint32_t ci, uint64_t item,
                                                 uint8_t *smem) {
  EncodeArgs a;
  a.values = c.values;
  a.n = c.n;
  a.bs = c.bs;
  a.nb = __ldg(B.prefix + ci + 1) - __ldg(B.prefix + ci);
  a.payload = c.payload;
  a.payload_cap = c.payload_cap;
  a.offsets = c.offsets;
  a.dir = c.dir;
  a.seq_models = nullptr;
  for (int i = 0; i < 10; ++i) a.polyX[i] = c.polyX[i];
  a.status = B.status + c.item0;
  a.ticket = nullptr;
  a.error = B.error;
  a.item_wait = 0;
  a.reversed = false;
  encode_rows_item<T, CODEC, 0, false>(a, item, c.rows, c.seq != 0, false, false, smem);
}

// Persistent encode: one ticket = one item of 256 / rows consecutive blocks of a column
// (which = 1: 512 threads, one block of 8193..16384 values).
template <int which>
__device__ __forceinline__ void batch_encode_items(const BatchArgs &B, uint8_t *smem) {
  __shared__ unsigned long long item;
  const uint64_t first = which ? B.enc_n[0] : 0, n = B.enc_n[which];
  for (;;) {
    if (threadIdx.x == 0) item = atomicAdd(B.ticket + 1 + which, 1ull);
    __syncthreads();
    const uint64_t it = item;
    __syncthreads();
    if (it >= n) break;
    const uint64_t e = __ldg(B.enc_items + first + it);
    const uint32_t ci = (uint32_t)(e >> 32);
    const DevCol &c = B.cols[ci];
    LECO_BATCH_DISPATCH(c.codec, c.dtype, batch_encode_one, B, c, ci, e & 0xffffffffull, smem);
    __syncthreads();  // shared memory is reused by the next item
  }
}
__global__ void __launch_bounds__(256, 3) batch_encode_kernel(BatchArgs B) {
  extern __shared__ __align__(256) uint8_t smem[];
  batch_encode_items<0>(B, smem);
}
__global__ void __launch_bounds__(512, 1) batch_encode_large_kernel(BatchArgs B) {
  extern __shared__ __align__(256) uint8_t smem[];
  batch_encode_items<1>(B, smem);
}

}  // namespace leco
