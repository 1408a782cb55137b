// leco_rows_kernel.cuh -- the single-column kernel of the row encoder, instantiated per value
// type in leco_rows_u32.cu and leco_rows_u64.cu.
#pragma once
#include "leco_rows.cuh"

namespace leco {

// The launch bounds of a kernel of up to NT threads: the CTAs per SM its registers are budgeted
// for are what the rows' shared memory allows (six of four warps with u64 LeCo rows, eight with
// u32 rows), capped at 1024 threads per SM.  NT = 448: blocks of nine to fourteen warps, two CTAs
// of the largest (degree-2: twelve warps, 80 registers) and three of nine warps.
template <typename T, int CODEC, int NT>
constexpr int rows_max_threads() { return NT != 448 ? NT : CODEC == kPoly2 ? 384 : sizeof(T) == 8 ? 448 : 512; }
template <typename T, int CODEC, int NT>
constexpr int rows_min_ctas() {
  if (NT == 448) return 2;
  if (sizeof(T) == 8) return CODEC == kPoly2 ? (NT == 128 ? 5 : NT == 256 ? 2 : 1) : (NT == 128 ? 6 : NT == 256 ? 3 : 1);
  if (CODEC == kPoly2) return NT == 128 ? 6 : NT == 256 ? 3 : 2;
  return CODEC == kLinear ? (NT == 128 ? 8 : NT == 256 ? 4 : 2) : (NT == 128 ? 10 : NT == 256 ? 5 : 2);
}

// One CTA of NT threads per item of NT / R blocks (RT: R, or 0: 32 and less), or with RT
// kWholeCta of R <= NT threads per block.  A column of one item needs no other; else CTA 0 is the
// publisher and CTA i + 1 takes item i (see the offsets in leco_rows.cuh).
template <typename T, int CODEC, int NT, uint32_t RT>
__global__ void __launch_bounds__(rows_max_threads<T, CODEC, NT>(), rows_min_ctas<T, CODEC, NT>())
    encode_rows_kernel(EncodeArgs a, uint32_t R, uint32_t items, bool ref) {
  extern __shared__ __align__(256) uint8_t smem_raw[];
  const bool alone = items == 1;
  const uint32_t role = a.reversed ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
  const bool again = !alone && role == 0;
  uint32_t item = alone ? 0 : role - 1;
  if (again) {
    const uint32_t head = publish_items<NT, RT != kWholeCta>(a.status, items, a.ticket + 1, a.error, smem_raw);
    if (!head) return;
    item = head - 1;
  }
  for (;;) {
    // the list goes on in the place of the item's first offset, which the item writes at its end
    uint32_t *next =
        reinterpret_cast<uint32_t *>(smem_raw + rows_layout(RT == kWholeCta ? R : NT, RT && RT != kWholeCta ? RT : R, sizeof(T), 0).next);
    if (again && threadIdx.x == 0) *next = (uint32_t)ld_relaxed(a.offsets + (uint64_t)item * ((RT == kWholeCta ? R : NT) / R));
    encode_rows_item<T, CODEC, RT, true>(a, item, R, ref, alone, again, smem_raw);
    if (!again) return;
    __syncthreads();
    if (!*next) return;
    item = *next - 1;
    __syncthreads();
  }
}

template <typename T, int CODEC, int NT, uint32_t RT>
int launch_rows_nt(const EncodeArgs &a, uint32_t R, bool ref, cudaStream_t st) {
  const uint32_t nt = RT == kWholeCta ? R : NT;
  const uint64_t nb_item = nt / R, items = (a.nb + nb_item - 1) / nb_item;
  const RowsLayout L = rows_layout(nt, R, sizeof(T), rows_sums(CODEC));
  const uint32_t smem = ref && !a.seq_models ? L.total : L.tab;
  // (the most a launch of this kernel takes: the limit belongs to the kernel)
  constexpr uint32_t most = rows_layout(NT, RT && RT != kWholeCta ? RT : RT ? NT : 8, sizeof(T), rows_sums(CODEC)).total;
  if (most > 48 * 1024) {
    const LaunchInfo i = launch_info<encode_rows_kernel<T, CODEC, NT, RT>>((int)nt, (int)most);
    if (i.error != cudaSuccess) return -(int)i.error;
  }
  encode_rows_kernel<T, CODEC, NT, RT><<<(unsigned)(items > 1 ? items + 1 : 1), nt, smem, st>>>(a, R, (uint32_t)items, ref);
  return 0;
}
template <typename T, int CODEC>
int launch_rows_t(const EncodeArgs &a, bool ref, cudaStream_t st) {
  const uint32_t R = column_rows_threads(CODEC, a.bs);
  switch (R) {
    case 64: return launch_rows_nt<T, CODEC, 128, 64>(a, R, ref, st);
    case 96: return launch_rows_nt<T, CODEC, 128, kWholeCta>(a, R, ref, st);
    case 128: return launch_rows_nt<T, CODEC, 128, 128>(a, R, ref, st);
    case 160:
    case 192: return launch_rows_nt<T, CODEC, 256, kWholeCta>(a, R, ref, st);
    case 256: return launch_rows_nt<T, CODEC, 256, 256>(a, R, ref, st);
    case 288:
    case 320:
    case 352:
    case 384:
    case 416:
    case 448: return launch_rows_nt<T, CODEC, 448, kWholeCta>(a, R, ref, st);
    case 512: return launch_rows_nt<T, CODEC, 512, 512>(a, R, ref, st);
    default: return launch_rows_nt<T, CODEC, 128, 0>(a, R, ref, st);
  }
}

}  // namespace leco
