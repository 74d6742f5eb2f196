// RMSNorm and reorder+RMSNorm for 16-bit rows with fp32 statistics.
//
// One CTA works on one row at a time and walks several rows; a thread owns the same one, two or four 16-byte chunks
// (8 values each) of every row, so that the weights can stay in registers, and the next row is on its way from memory
// while the current one is reduced, scaled and stored (one barrier per row).  Wide rows of matrices beyond the L2 take one
// CTA each (rmsnorm_row_kernel), rows of more than 32768 values (of a sum: 16384) are read twice.  Bound by HBM: 16384 x
// 4096 bf16 takes 43.5 us (6.17 TB/s) where one CTA per row, with nothing in flight while it reduced, took 63.0; 37 x
// 8000 fp16 takes 2.2 us where it took 3.1; a single launch of 4096 x 8192 bf16 on a cold L2 28.7 where it took 30.7.
// Tile order reads at 2048 x 8192 behind its GEMM: 54.3 us for the pair against 57.2 with the tile found anew for every
// load.  With a sum (two rows in, two out) 2048 x 4096 bf16 takes 9.8 us.  Unlike the reference kernels (reference: src/rmsnorm/rmsnorm.cuh:12-115, block size dim/16, eps fixed to
// 1e-5, default stream) any dim % 8 == 0 works, eps is an argument and the launch goes to the caller's stream.
#include "rmsnorm.h"

#include "gemm_fused_sm100.cuh"

namespace fo {

namespace {

constexpr int kMaxNormThreads = 1024;
constexpr int kRowThreads = 256;  // rmsnorm_row_kernel
constexpr int kRowChunks = 8;

// What a row is before it is normalised: as stored, stored in tile order, or the sum of two rows (written back).
enum NormInput { NORM_ROWS, NORM_TILES, NORM_SUM };

template <bool BF16>
__device__ __forceinline__ uint32_t add2(uint32_t a, uint32_t b) {
  const float2 f = unpack2<BF16>(a), g = unpack2<BF16>(b);
  return pack2<BF16>(f.x + g.x, f.y + g.y);
}
template <bool BF16>
__device__ __forceinline__ uint4 add_chunk(const uint4& a, const uint4& b) {
  return make_uint4(add2<BF16>(a.x, b.x), add2<BF16>(a.y, b.y), add2<BF16>(a.z, b.z), add2<BF16>(a.w, b.w));
}

// Eight values as floats that stay in registers (the compiler would rather unpack them again).
template <bool BF16>
__device__ __forceinline__ void unpack_chunk(float (&f)[8], const uint4& v) {
  const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 p = unpack2<BF16>(u[i]);
    f[2 * i] = p.x;
    f[2 * i + 1] = p.y;
    asm volatile("" : "+f"(f[2 * i]), "+f"(f[2 * i + 1]));
  }
}

// `r` and `sum`: NORM_SUM only.
template <bool BF16, int INPUT, int CPT>
__global__ void __launch_bounds__(kMaxNormThreads) rmsnorm_kernel(const uint16_t* x, const uint16_t* r, uint16_t* sum,
                                                                  uint16_t* out, const uint16_t* __restrict__ w,
                                                                  int rows, int dim, float eps, OutLayout L) {
  constexpr bool ADD = INPUT == NORM_SUM;
  __shared__ float red[2][kMaxNormThreads / 32];
  ptx::wait_for_previous_kernel();
  ptx::allow_next_kernel();
  const int n_chunks = dim >> 3;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int warps = blockDim.x >> 5;

  // Tile order: a thread's columns lie in the same tile column, at the same place in it, in every row.
  int tile_col[INPUT == NORM_TILES ? CPT : 1], in_tile[INPUT == NORM_TILES ? CPT : 1];
  if constexpr (INPUT == NORM_TILES) {
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
      const int col = min(static_cast<int>(threadIdx.x + k * blockDim.x), n_chunks - 1) * 8;
      tile_col[k] = col / L.bn;
      in_tile[k] = col - tile_col[k] * L.bn;
    }
  }
  auto load = [&](int row, uint4 (&v)[CPT], uint4 (&a)[ADD ? CPT : 1]) {
    [[maybe_unused]] const int tile_row = INPUT == NORM_TILES ? row / L.bm : 0;
    [[maybe_unused]] const int row_in_tile = INPUT == NORM_TILES ? row - tile_row * L.bm : 0;
    [[maybe_unused]] int slot[INPUT == NORM_TILES ? CPT : 1];
    if constexpr (INPUT == NORM_TILES) {
#pragma unroll
      for (int k = 0; k < CPT; ++k) {
        slot[k] = tile_row * L.tn + tile_col[k];
        if (L.ra != nullptr) slot[k] = __ldg(L.ra + slot[k]);
      }
    }
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
      // a chunk past the end of the row is clamped and its value dropped: the loads stay unconditional and go out together
      const int c = min(static_cast<int>(threadIdx.x + k * blockDim.x), n_chunks - 1);
      const uint16_t* src;
      if constexpr (INPUT == NORM_TILES) {
        int view = slot[k], place = 0;  // tile row of the view and place in it
        if (L.rldn > 1) {
          view = slot[k] / L.rldn;
          place = slot[k] - view * L.rldn;
        }
        src = x + (static_cast<long long>(view) * L.bm + row_in_tile) * (static_cast<long long>(L.rldn) * L.bn) +
              place * L.bn + in_tile[k];
      } else src = x + static_cast<long long>(row) * dim + c * 8;
      v[k] = *reinterpret_cast<const uint4*>(src);
      if constexpr (ADD) a[k] = *reinterpret_cast<const uint4*>(r + static_cast<long long>(row) * dim + c * 8);
    }
  };

  // room for the weights beside two rows; four chunks (two of a sum) read them from L1 for each row
  constexpr bool KEEP = CPT <= (ADD ? 1 : 2);
  const uint4* weights = reinterpret_cast<const uint4*>(w);
  uint4 v[CPT], a[ADD ? CPT : 1], g[KEEP ? CPT : 1];
  // unsigned: the last step of a CTA may pass the largest int (rows of 8 values can be that many)
  const unsigned n_rows = rows;
  unsigned row = blockIdx.x;
  load(row, v, a);
  if constexpr (KEEP) {
#pragma unroll
    for (int k = 0; k < CPT; ++k) g[k] = __ldg(weights + min(static_cast<int>(threadIdx.x + k * blockDim.x), n_chunks - 1));
  }
  for (int par = 0; row < n_rows; par ^= 1) {
    float ssq = 0.f;
    if constexpr (ADD) {
      uint4* dst = reinterpret_cast<uint4*>(sum + static_cast<long long>(row) * dim);
#pragma unroll
      for (int k = 0; k < CPT; ++k) {
        const int c = threadIdx.x + k * blockDim.x;
        v[k] = add_chunk<BF16>(v[k], a[k]);
        if (c < n_chunks) dst[c] = v[k];
      }
    }
    // Up to two chunks (one of a sum, whose two would not fit) stay unpacked between the statistics and the scaling: less
    // follows the barrier, and with these registers no CTA of the next grid finds a place before one of this grid has ended
    // (with five of them on some SMs the grid ended later).  That takes more than 48 registers a thread with two chunks (55 as
    // compiled, 58 in tile order; a fifth CTA of 256 threads fits at 48): a build with fewer would be slower, not wrong.
    // Launch after launch, fp16: 16384 x 4096 49.0 -> 43.5 us, 2048 x
    // 4096 7.5 -> 5.2, 1000 x 1024 2.5 -> 2.1; in tile order 4096 x 9216 39.9 -> 36.7, 2048 x 8192 12.9 -> 12.3.
    constexpr bool UNPACKED = INPUT == NORM_SUM ? CPT == 1 : CPT <= 2;
    float f[UNPACKED ? CPT : 1][8];
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
      if constexpr (UNPACKED) {
        unpack_chunk<BF16>(f[k], v[k]);
        float q = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) q += f[k][e] * f[k][e];
        ssq += static_cast<int>(threadIdx.x + k * blockDim.x) < n_chunks ? q : 0.f;
      } else {
        ssq += static_cast<int>(threadIdx.x + k * blockDim.x) < n_chunks ? sum_squares<BF16>(v[k]) : 0.f;
      }
    }
    const unsigned next = row + gridDim.x;
    uint4 nv[CPT];
    if (next < n_rows) load(next, nv, a);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ssq += __shfl_xor_sync(0xffffffffu, ssq, o);
    if (warps > 1) {
      if (lane == 0) red[par][warp] = ssq;  // two sets alternate: one barrier per row is enough
      __syncthreads();
      ssq = lane < warps ? red[par][lane] : 0.f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ssq += __shfl_xor_sync(0xffffffffu, ssq, o);
    }
    const float rstd = rsqrtf(ssq / static_cast<float>(dim) + eps);
    uint4* dst = reinterpret_cast<uint4*>(out + static_cast<long long>(row) * dim);
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
      const int c = threadIdx.x + k * blockDim.x;
      const uint4 w4 = KEEP ? g[KEEP ? k : 0] : __ldg(weights + min(c, n_chunks - 1));
      if constexpr (UNPACKED) {
        if (c < n_chunks) {
          dst[c] = make_uint4(norm_pack2<BF16>(f[k][0], f[k][1], rstd, w4.x), norm_pack2<BF16>(f[k][2], f[k][3], rstd, w4.y),
                              norm_pack2<BF16>(f[k][4], f[k][5], rstd, w4.z), norm_pack2<BF16>(f[k][6], f[k][7], rstd, w4.w));
        }
      } else {
        if (c < n_chunks) dst[c] = scale_chunk<BF16>(v[k], rstd, w4);
      }
    }
#pragma unroll
    for (int k = 0; k < CPT; ++k) v[k] = nv[k];
    row = next;
  }
}

// Rows as stored, of up to 16384 values, one CTA of 256 threads per row: five rows of an SM are loaded, reduced and stored
// independently of one another.  For matrices that stream through HBM (see launch_typed).
template <bool BF16>
__global__ void __launch_bounds__(kRowThreads, 5) rmsnorm_row_kernel(const uint16_t* x, uint16_t* out,
                                                                     const uint16_t* __restrict__ w, int dim, float eps) {
  __shared__ float red[kRowThreads / 32];
  const int n_chunks = dim >> 3;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long row_off = static_cast<long long>(blockIdx.x) * dim;
  const uint4* src = reinterpret_cast<const uint4*>(x + row_off);
  uint4 v[kRowChunks];
#pragma unroll
  for (int k = 0; k < kRowChunks; ++k) v[k] = src[min(static_cast<int>(threadIdx.x) + k * kRowThreads, n_chunks - 1)];
  float ssq = 0.f;
#pragma unroll
  for (int k = 0; k < kRowChunks; ++k) {
    if (static_cast<int>(threadIdx.x) + k * kRowThreads < n_chunks) ssq += sum_squares<BF16>(v[k]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ssq += __shfl_xor_sync(0xffffffffu, ssq, o);
  if (lane == 0) red[warp] = ssq;
  __syncthreads();
  ssq = 0.f;
#pragma unroll
  for (int i = 0; i < kRowThreads / 32; ++i) ssq += red[i];
  const float rstd = rsqrtf(ssq / static_cast<float>(dim) + eps);
  uint4* dst = reinterpret_cast<uint4*>(out + row_off);
#pragma unroll
  for (int k = 0; k < kRowChunks; ++k) {
    const int c = static_cast<int>(threadIdx.x) + k * kRowThreads;
    if (c < n_chunks) dst[c] = scale_chunk<BF16>(v[k], rstd, __ldg(reinterpret_cast<const uint4*>(w) + c));
  }
}

// Rows wider than the registers of a CTA hold: one CTA per row, read twice.
template <bool BF16, int INPUT>
__global__ void __launch_bounds__(kMaxNormThreads) rmsnorm_wide_kernel(const uint16_t* x, const uint16_t* r,
                                                                       uint16_t* sum, uint16_t* out,
                                                                       const uint16_t* __restrict__ w, int dim,
                                                                       float eps, OutLayout L) {
  __shared__ float red[kMaxNormThreads / 32];
  ptx::wait_for_previous_kernel();
  ptx::allow_next_kernel();
  const int row = blockIdx.x;
  const int n_chunks = dim >> 3;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long row_off = static_cast<long long>(row) * dim;
  if constexpr (INPUT == NORM_SUM) {  // every thread reads back exactly the chunks it wrote
    for (int c = threadIdx.x; c < n_chunks; c += kMaxNormThreads) {
      reinterpret_cast<uint4*>(sum + row_off)[c] = add_chunk<BF16>(reinterpret_cast<const uint4*>(x + row_off)[c],
                                                                   reinterpret_cast<const uint4*>(r + row_off)[c]);
    }
  }
  auto src_ptr = [&](int c) -> const uint4* {
    if constexpr (INPUT == NORM_SUM) return reinterpret_cast<const uint4*>(sum + row_off) + c;
    else if constexpr (INPUT == NORM_TILES) return reinterpret_cast<const uint4*>(x + layout_offset(L, row, c * 8));
    else return reinterpret_cast<const uint4*>(x + row_off) + c;
  };
  float ssq = 0.f;
  for (int c = threadIdx.x; c < n_chunks; c += kMaxNormThreads) ssq += sum_squares<BF16>(*src_ptr(c));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ssq += __shfl_xor_sync(0xffffffffu, ssq, o);
  if (lane == 0) red[warp] = ssq;
  __syncthreads();
  ssq = red[lane];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ssq += __shfl_xor_sync(0xffffffffu, ssq, o);
  const float rstd = rsqrtf(ssq / static_cast<float>(dim) + eps);
  uint4* dst = reinterpret_cast<uint4*>(out + row_off);
  for (int c = threadIdx.x; c < n_chunks; c += kMaxNormThreads) {
    dst[c] = scale_chunk<BF16>(*src_ptr(c), rstd, __ldg(reinterpret_cast<const uint4*>(w) + c));
  }
}

// Launch whose CTAs may be placed while the kernel before it drains (they wait for it themselves).
template <typename... Params, typename... Args>
cudaError_t launch_after(void (*kernel)(Params...), int grid, int threads, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(grid), 1, 1);
  cfg.blockDim = dim3(static_cast<unsigned>(threads), 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

template <bool BF16, int INPUT>
cudaError_t launch_typed(const uint16_t* x, const uint16_t* r, uint16_t* sum, uint16_t* out, const uint16_t* w, int rows,
                         int dim, float eps, const OutLayout& L, cudaStream_t stream) {
  const int n_chunks = dim >> 3;
  // A sum of more than two chunks per thread does not fit the registers beside the next row (the kernel spills):
  // 4096 x 20480 bf16 takes 154 us in that form, 113 here, 137 as an addition and an RMSNorm of their own.
  if (n_chunks > (INPUT == NORM_SUM ? 2 : 4) * kMaxNormThreads) {
    return launch_after(rmsnorm_wide_kernel<BF16, INPUT>, rows, kMaxNormThreads, stream, x, r, sum, out, w, dim, eps, L);
  }
  const int sms = device_sm_count();
  // Few rows (up to two per SM): as many threads per row as it has chunks, since only the latency of one row counts.
  // Many rows: two chunks per thread, which leaves fewer warps to wait at the row's barrier and keeps the weights in
  // registers; four need the registers of the weights (the kernel spills at 64 a thread) and serve wide rows only.
  int cpt = rows <= 2 * sms || n_chunks <= 32 ? 1 : 2;
  while (n_chunks > cpt * kMaxNormThreads) cpt *= 2;
  if constexpr (INPUT == NORM_ROWS) {
    // Past the L2 (126 MB) the matrix streams, and CTAs that do not wait for one another keep HBM busier than few large ones
    // that walk: 8192 x 12288 bf16 74.8 -> 64.7 us, 24576 x 6144 116 -> 96, 24576 x 8192 130 -> 121.  Rows of up to 5120
    // values leave most of the registers of such a CTA empty (24576 x 5120: 83 us walked, 100 one by one).
    if (cpt == 2 && n_chunks > 640 && 2.0 * rows * dim >= 126e6) {
      rmsnorm_row_kernel<BF16><<<rows, kRowThreads, 0, stream>>>(x, out, w, dim, eps);
      return cudaGetLastError();
    }
    // More than 8192 values: with two chunks per thread a single CTA fits an SM and nothing runs while it waits at its
    // barrier.  From ten rows per SM on, four chunks and two or three CTAs: 4096 x 9216 32.5 -> 27.1 us, 2048 x 16384 24.8 ->
    // 23.9; with fewer rows two chunks are the faster form (1024 x 16384 13.7 us against 15.1).
    if (cpt == 2 && n_chunks > kMaxNormThreads && rows > 10 * sms) cpt = 4;
  }
  const int threads = ((n_chunks + cpt - 1) / cpt + 31) / 32 * 32;
  // 64 registers a thread: the CTAs that are resident together
  int per_sm = kMaxNormThreads / threads;
  if (per_sm > 32) per_sm = 32;
  const int grid = rows < sms * per_sm ? rows : sms * per_sm;
  auto kernel = cpt == 1 ? rmsnorm_kernel<BF16, INPUT, 1> : rmsnorm_kernel<BF16, INPUT, 2>;
  if constexpr (INPUT != NORM_SUM) {
    if (cpt == 4) kernel = rmsnorm_kernel<BF16, INPUT, 4>;
  }
  return launch_after(kernel, grid, threads, stream, x, r, sum, out, w, rows, dim, eps, L);
}

template <int INPUT>
cudaError_t launch(const void* x, const void* r, void* sum, void* out, const void* w, int rows, int dim, float eps,
                   const OutLayout& L, DType dt, cudaStream_t stream) {
  if (rows <= 0 || dim <= 0 || dim % 8 != 0) return cudaErrorInvalidValue;
  // the kernels load and store 16 bytes at a time
  auto address = [](const void* p) { return reinterpret_cast<uintptr_t>(p); };
  if ((address(x) | address(r) | address(sum) | address(out) | address(w)) & 15u) return cudaErrorMisalignedAddress;
  auto typed = dt == DT_BF16 ? launch_typed<true, INPUT> : launch_typed<false, INPUT>;
  return typed(static_cast<const uint16_t*>(x), static_cast<const uint16_t*>(r), static_cast<uint16_t*>(sum),
               static_cast<uint16_t*>(out), static_cast<const uint16_t*>(w), rows, dim, eps, L, stream);
}

}  // namespace

cudaError_t launch_rmsnorm(const void* x, void* out, const void* w, int rows, int dim, float eps, DType dt,
                           cudaStream_t stream) {
  return launch<NORM_ROWS>(x, nullptr, nullptr, out, w, rows, dim, eps, OutLayout{}, dt, stream);
}

cudaError_t launch_reorder_rmsnorm(const void* x, void* out, const void* w, int rows, int dim, float eps,
                                   const OutLayout& in_layout, DType dt, cudaStream_t stream) {
  // the kernel finds its tiles itself: no natural layout (bn = 0) and no row map
  if (!in_layout.tiled || in_layout.row_map != nullptr || in_layout.bn <= 0 || in_layout.bn % 8 != 0 ||
      in_layout.bm <= 0 || in_layout.rldn <= 0) {
    return cudaErrorInvalidValue;
  }
  return launch<NORM_TILES>(x, nullptr, nullptr, out, w, rows, dim, eps, in_layout, dt, stream);
}

cudaError_t launch_add_rmsnorm(const void* x, const void* r, void* sum, void* out, const void* w, int rows, int dim,
                               float eps, DType dt, cudaStream_t stream) {
  return launch<NORM_SUM>(x, r, sum, out, w, rows, dim, eps, OutLayout{}, dt, stream);
}

}  // namespace fo
