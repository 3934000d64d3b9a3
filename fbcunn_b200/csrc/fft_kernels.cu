// Batched 2-D R2C / C2R FFT kernels (sm_100a): one thread block transforms a tile
// of T planes that are neighbours in the spectrum's innermost index, entirely in
// shared memory and registers, and writes / reads the bin-major spectrum in runs of
// T complex values.  Phases and index arithmetic live in fft_core.cuh.
//
// Stands where the reference launches fbfft2D / fbifft2D
// (src/fft/FBFFTHost.cpp:84-111); unlike the reference's sizes 64 and 128
// (two launches through a transposed global buffer, :56-104) every size is a
// single launch with no global scratch.
#include <atomic>
#include <cstdlib>
#include <mutex>
#include <vector>

#include "kernels.h"

namespace fbfft {

// The opt-in to a kernel's dynamic shared memory is per device and function and only ever grows:
// it is asked for when a launch needs more than any launch of that kernel on that device before.
cudaError_t ensure_dynamic_smem(const void* kernel, int bytes) {
  struct Entry {
    const void* kernel;
    int device, bytes;
  };
  static std::mutex mutex;
  static std::vector<Entry> seen;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
  std::lock_guard<std::mutex> lock(mutex);
  for (Entry& e : seen)
    if (e.kernel == kernel && e.device == dev) {
      if (e.bytes >= bytes) return cudaSuccess;
      cudaError_t r = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
      if (r == cudaSuccess)
        e.bytes = bytes;
      else
        cudaGetLastError();
      return r;
    }
  cudaError_t r = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (r == cudaSuccess)
    seen.push_back(Entry{kernel, dev, bytes});
  else
    cudaGetLastError();
  return r;
}

namespace {

std::atomic<uint64_t> g_launches{0};

constexpr int kRowSumWarpLimit = 512;  // values a single warp sums (16 a lane, all in flight at once)

template <int N, int T>
constexpr int block_threads() {
  return ((N / 2 + 1) * T + 31) / 32 * 32 < 64 ? 64 : ((N / 2 + 1) * T + 31) / 32 * 32;
}

// dst[r] (=|+=) scale * sum of a row: a warp per row, or -- long rows -- the block per row.
__device__ void row_sum_block(const RowSum& s, int block, char* smem) {
  const bool per_warp = s.count <= kRowSumWarpLimit;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int row = per_warp ? block * nwarps + warp : block;
  float v = 0.f;
  if (row < s.rows)
    for (int i = per_warp ? lane : (int)threadIdx.x; i < s.count; i += per_warp ? 32 : (int)blockDim.x)
      v += s.src[row * s.ld + i * s.step];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (!per_warp) {
    float* part = reinterpret_cast<float*>(smem);
    if (lane == 0) part[warp] = v;
    __syncthreads();
    v = 0.f;
    if (threadIdx.x == 0)
      for (int i = 0; i < nwarps; ++i) v += part[i];
  }
  if (row < s.rows && (per_warp ? lane == 0 : threadIdx.x == 0))
    s.dst[row] = s.accumulate ? s.dst[row] + s.scale * v : s.scale * v;
}
int row_sum_blocks(const RowSum& s, int threads) {
  const int rows_per_block = s.count <= kRowSumWarpLimit ? threads / 32 : 1;
  return (s.rows + rows_per_block - 1) / rows_per_block;
}

// One launch transforms the planes of up to OPS operands of a pass (its two or three real tensors, or the
// two spectra that a backward call inverts): the block index runs over the tiles of all of them.  Small
// layers are bound by launches, and a small operand next to a large one would leave most SMs idle in a
// launch of its own.  With OPS = 1 the parameters are compile-time addresses in the constant bank.
template <int OPS>
struct FftBatch {
  FftParams p[OPS];
  FftGeom g[OPS];
  int tiles_x[OPS];    // tiles along the inner index
  int tile_end[OPS];   // running total of tiles
  int sum_blocks;      // inverse only: leading blocks that do `sum` instead of a tile
  RowSum sum;
};

// Runs body(params, geometry, tile inside the operand, tiles along the inner index) for the operand that
// `tile` belongs to.  The body is instantiated once per operand: with the operand's number known at compile
// time its parameters stay operands of the instructions, where a run-time index cost 10 % (32 points, plain
// instruction issue) and 16 registers (16 points).
template <int OPS, class Body>
__device__ __forceinline__ void with_operand(const FftBatch<OPS>& b, int tile, Body body) {
  if constexpr (OPS == 1) {
    body(b.p[0], b.g[0], tile, b.tiles_x[0]);
  } else {
    if (tile < b.tile_end[0])
      body(b.p[0], b.g[0], tile, b.tiles_x[0]);
    else if (OPS == 2 || tile < b.tile_end[1])
      body(b.p[1], b.g[1], tile - b.tile_end[0], b.tiles_x[1]);
    else if constexpr (OPS > 2)
      body(b.p[2], b.g[2], tile - b.tile_end[1], b.tiles_x[2]);
  }
}

// MODE: planes of some operand are tiles of images, or the spectrum is the reference's tensor (kernels of their
// own, so that the others stay as they are).
template <int N, int T, int OPS, int MODE>
__global__ void __launch_bounds__(block_threads<N, T>())
fft2d_forward_kernel(const __grid_constant__ FftBatch<OPS> b) {
  extern __shared__ __align__(16) char smem[];
  const int tid = threadIdx.x;
  grid_dependency_wait();
  with_operand(b, blockIdx.x, [&](const FftParams& p, const FftGeom& g, int tile, int tiles_x) {
    const int row = tile / tiles_x;
    const int inner0 = (tile - row * tiles_x) * T;
    Forward<N, T>::template load<MODE>(p, g, smem, tid, blockDim.x, row, inner0);
    __syncthreads();
    LineRegs<N> regs;
    Forward<N, T>::template row_fetch<MODE>(p, g, smem, tid, row, inner0, regs);
    __syncthreads();  // the column buffer aliases the staged planes
    Forward<N, T>::row_pass(g, smem, tid, regs);
    __syncthreads();
    Forward<N, T>::template col_pass<MODE>(p, g, smem, tid, row, inner0);
  });
}

template <int N, int T, int OPS, int MODE>
__global__ void __launch_bounds__(block_threads<N, T>())
fft2d_inverse_kernel(const __grid_constant__ FftBatch<OPS> b) {
  extern __shared__ __align__(16) char smem[];
  const int tid = threadIdx.x;
  grid_dependency_wait();
  if ((int)blockIdx.x < b.sum_blocks) {
    row_sum_block(b.sum, blockIdx.x, smem);
    return;
  }
  with_operand(b, (int)blockIdx.x - b.sum_blocks, [&](const FftParams& p, const FftGeom& g, int tile, int tiles_x) {
    const int row = tile / tiles_x;
    const int inner0 = (tile - row * tiles_x) * T;
    Inverse<N, T>::template col_pass<MODE>(p, g, smem, tid, row, inner0);
    __syncthreads();
    LineRegs<N> regs;
    Inverse<N, T>::row_fetch(g, smem, tid, regs);
    __syncthreads();  // the staged output aliases the column buffer
    Inverse<N, T>::template row_pass<MODE>(p, g, smem, tid, row, inner0, regs);
    __syncthreads();
    Inverse<N, T>::template store<MODE>(p, g, smem, tid, blockDim.x, row, inner0);
  });
}

__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// The cooperative kernels look the operand up per tile: `tile` becomes the tile's number inside the operand.
template <int OPS>
__device__ __forceinline__ int operand_of_tile(const FftBatch<OPS>& b, int& tile) {
  if constexpr (OPS == 1) {
    return 0;
  } else {
    int op = 0;
#pragma unroll
    for (int i = 1; i < OPS; ++i)
      if (tile >= b.tile_end[i - 1]) op = i;
    if (op > 0) tile -= b.tile_end[op - 1];
    return op;
  }
}

// PM: the spectra are plane-major (bins contiguous), else bin-major.
template <int N, int T, int OPS, bool PM>
__global__ void __launch_bounds__(coop_shape(N, false, PM).threads, coop_shape(N, false, PM).blocks)
fft2d_forward_coop_kernel(const __grid_constant__ FftBatch<OPS> b) {
  extern __shared__ __align__(16) char smem[];
  const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const int total = b.tile_end[OPS - 1];
  grid_dependency_wait();
  // persistent blocks: tile w, then w + gridDim.x, ...; the real planes of the next tile are
  // pulled into L2 while this one is transformed (CoopShape::persistent; else a block has one tile)
  for (int w = blockIdx.x; w < total; w += gridDim.x) {
  int tile = w;
  const int op = operand_of_tile(b, tile);
  const FftParams& p = b.p[op];
  const FftGeom& g = b.g[op];
  const int tiles_x = b.tiles_x[op];
  const int row = tile / tiles_x;
  const int inner0 = (tile - row * tiles_x) * T;
  if (tile + (int)gridDim.x < tiles_x * p.n_rows) {
    const int wn = tile + gridDim.x;
    const int rown = wn / tiles_x, innern = (wn - rown * tiles_x) * T;
    const long long plane_bytes = (long long)p.h * p.w * 4;
    for (int t = 0; t < T; ++t) {
      if (innern + t >= p.n_inner) break;
      const char* src = reinterpret_cast<const char*>(p.real_in) +
                        (rown * p.real_row_stride + (innern + t) * p.real_inner_stride) * plane_bytes;
      for (long long off = (long long)tid * 128; off < plane_bytes; off += (long long)nth * 128) prefetch_l2(src + off);
    }
  }
  using F = CoopForward<N, T>;
  {
    const bool half = F::L::half_tasks(g, nth);
    const int task = half ? F::L::TASK_LINES / 2 : F::L::TASK_LINES;
    float2 tw[F::N1];  // a lane meets the same n2 in all its items
    F::row_twiddles(lane, tw);
    for (int line0 = warp * task; line0 < g.lines1; line0 += (nth >> 5) * task) {
      F::row_step1(p, g, smem, lane, row, inner0, line0, tw, half);
      __syncwarp();
      // groups of eight lanes hold the eight residues of one line; mirror residues are
      // neighbours, so one shuffle hands each lane the partner's odd-indexed outputs
#pragma unroll 1
      for (int item = lane; item < task * F::N1; item += 32) {
        float2 u[F::N2], mirror_odd[F::N2 / 2];
        const bool active = F::row_step2_fft(g, smem, line0, item, u);
#pragma unroll
        for (int i = 0; i < F::N2 / 2; ++i) {  // every lane takes part: the reads above are over after this
          mirror_odd[i].x = __shfl_xor_sync(0xffffffffu, u[2 * i + 1].x, 1);
          mirror_odd[i].y = __shfl_xor_sync(0xffffffffu, u[2 * i + 1].y, 1);
        }
        __syncwarp();
        if (active) F::row_step2_split(g, smem, line0, item, u, mirror_odd);
      }
    }
  }
  __syncthreads();
  CoopForward<N, T>::col_step1(g, smem, tid, nth);
  __syncthreads();
  CoopForward<N, T>::template col_step2<PM>(p, g, smem, tid, nth, row, inner0);
  __syncthreads();  // the buffers are reused by the next tile
  }
}

template <int N, int T, int OPS, bool PM>
__global__ void __launch_bounds__(coop_shape(N, true, PM).threads, coop_shape(N, true, PM).blocks)
fft2d_inverse_coop_kernel(const __grid_constant__ FftBatch<OPS> b) {
  extern __shared__ __align__(16) char smem[];
  const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const int total = b.tile_end[OPS - 1];
  grid_dependency_wait();
  const int first = (int)blockIdx.x - b.sum_blocks, step = (int)gridDim.x - b.sum_blocks;
  if (first < 0) {
    row_sum_block(b.sum, blockIdx.x, smem);
    return;
  }
  for (int w = first; w < total; w += step) {
  int tile = w;
  const int op = operand_of_tile(b, tile);
  const FftParams& p = b.p[op];
  const FftGeom& g = b.g[op];
  const int tiles_x = b.tiles_x[op];
  const int row = tile / tiles_x;
  const int inner0 = (tile - row * tiles_x) * T;
  if (PM && tile + step < tiles_x * p.n_rows) {  // plane-major: the next tile's spectra are contiguous
    const int wn = tile + step;
    const int rown = wn / tiles_x, innern = (wn - rown * tiles_x) * T;
    const long long plane_bytes = (long long)(N / 2 + 1) * N * 8;
    for (int t = 0; t < T; ++t) {
      if (innern + t >= p.n_inner) break;
      const char* src = reinterpret_cast<const char*>(p.spec + rown * p.spec_row + (innern + t) * p.spec_inner);
      for (long long off = (long long)tid * 128; off < plane_bytes; off += (long long)nth * 128) prefetch_l2(src + off);
    }
  }
  CoopInverse<N, T>::template col_step1<PM>(p, g, smem, tid, nth, row, inner0);
  __syncthreads();
  CoopInverse<N, T>::col_step2(g, smem, tid, nth);
  __syncthreads();
  using I = CoopInverse<N, T>;
  {
    const bool half = I::L::half_tasks(g, nth);
    const int task = half ? I::L::TASK_LINES / 2 : I::L::TASK_LINES;
    float2 tw[I::N1];  // a lane meets the same n2 in all its items
    I::row_twiddles(lane, tw);
    for (int line0 = warp * task; line0 < g.lines1; line0 += (nth >> 5) * task) {
      float2 v0[I::N1], v1[I::N1];
      const bool on0 = I::row_step1_fft(p, g, smem, line0, lane, v0);
      const bool on1 = !half && I::row_step1_fft(p, g, smem, line0, lane + 32, v1);
      __syncwarp();
      if (on0) I::row_step1_store(p, g, smem, line0, lane, v0, tw);
      if (on1) I::row_step1_store(p, g, smem, line0, lane + 32, v1, tw);
      __syncwarp();
#pragma unroll 1
      for (int item = lane; item < task * I::N1; item += 32) I::row_step2(p, g, smem, row, inner0, line0, item);
    }
  }
  __syncthreads();  // mid is rewritten by the next tile
  }
}

// ---- batched 1-D transforms up to 32 points: the row phases of the thread-per-line kernels (larger
// ---- sizes have kernels of their own, fft1d_lines.cu)
template <int N, int T>
__global__ void __launch_bounds__(block_threads<N, T>())
fft1d_forward_kernel(const __grid_constant__ FftParams p, const __grid_constant__ FftGeom g) {
  static_assert(N <= 32, "thread-per-line sizes");
  extern __shared__ __align__(16) char smem[];
  const int tid = threadIdx.x, nth = blockDim.x;
  const int inner0 = blockIdx.x * T;
  grid_dependency_wait();
  Forward<N, T>::load(p, g, smem, tid, nth, 0, inner0);
  __syncthreads();
  LineRegs<N> regs;
  Forward<N, T>::row_fetch(p, g, smem, tid, 0, inner0, regs);
  __syncthreads();
  Forward<N, T>::row_pass(g, smem, tid, regs);
  __syncthreads();
  Rows1D<N, T>::store_spectrum(p, g, smem, tid, nth, inner0);
}

template <int N, int T>
__global__ void __launch_bounds__(block_threads<N, T>())
fft1d_inverse_kernel(const __grid_constant__ FftParams p, const __grid_constant__ FftGeom g) {
  static_assert(N <= 32, "thread-per-line sizes");
  extern __shared__ __align__(16) char smem[];
  const int tid = threadIdx.x, nth = blockDim.x;
  const int inner0 = blockIdx.x * T;
  grid_dependency_wait();
  Rows1D<N, T>::load_spectrum(p, g, smem, tid, nth, inner0);
  __syncthreads();
  LineRegs<N> regs;
  Inverse<N, T>::row_fetch(g, smem, tid, regs);
  __syncthreads();
  Inverse<N, T>::row_pass(p, g, smem, tid, 0, inner0, regs);
  __syncthreads();
  Inverse<N, T>::store(p, g, smem, tid, nth, 0, inner0);
}

// Blocks of a cooperative kernel: persistent ones as many as are resident at once.
long long coop_grid(const CoopShape& shape, long long tiles) {
  const long long resident = (long long)sm_count() * shape.blocks;
  return shape.persistent && tiles > resident ? resident : tiles;
}

template <int N, int T, int OPS, bool INVERSE, bool PM>
constexpr auto coop_kernel() {
  constexpr CoopShape shape = coop_shape(N, INVERSE, PM);
  static_assert(shape.threads % 32 == 0, "whole warps");
  static_assert(shape.blocks * (N * CoopLayout<N, T>::PITCH2 * 8 + 1024) <= 228 * 1024, "shared memory of an SM");
  if constexpr (INVERSE)
    return fft2d_inverse_coop_kernel<N, T, OPS, PM>;
  else
    return fft2d_forward_coop_kernel<N, T, OPS, PM>;
}
template <int N, int T, int OPS, bool INVERSE, int MODE>
constexpr auto line_kernel() {
  if constexpr (INVERSE)
    return fft2d_inverse_kernel<N, T, OPS, MODE>;
  else
    return fft2d_forward_kernel<N, T, OPS, MODE>;
}

// The kernels address the spectrum with 32-bit element offsets.
bool spectrum_fits(const FftParams& p, int N) {
  const long long bins = (long long)(N / 2 + 1) * N;
  return bins * p.n_rows * p.kc < (1LL << 31);
}

template <int N, int OPS, bool INVERSE>
cudaError_t run_batch(const FftParams* ops, int count, const RowSum* sum, cudaStream_t stream) {
  constexpr int T = fft_tile(N);
  FftBatch<OPS> b{};
  long long tiles = 0;
  int smem = 0;
  int mode = kPlanes;
  const bool plane_major = ops[0].spec_bin == 1;
  for (int i = 0; i < OPS; ++i) {
    if (i < count) {
      if ((ops[i].spec_bin == 1) != plane_major) return cudaErrorInvalidConfiguration;
      b.p[i] = ops[i];
      if (ops[i].view.nw) mode = kTiles;
      if (ops[i].reference) mode = kReference;
      b.g[i] = INVERSE ? inverse_geom(N, T, ops[i].h, ops[i].w, plane_major)
                       : forward_geom(N, T, ops[i].h, ops[i].w, ops[i].off_y, ops[i].off_x, plane_major);
      b.tiles_x[i] = ((INVERSE ? ops[i].n_inner : ops[i].kc) + T - 1) / T;
      tiles += (long long)b.tiles_x[i] * ops[i].n_rows;
      if (b.g[i].smem_bytes > smem) smem = b.g[i].smem_bytes;
    }
    b.tile_end[i] = (int)tiles;
  }
  if (tiles > 0x7fffffff) return cudaErrorInvalidConfiguration;
  const int threads = b.g[0].threads;
  if (sum && sum->rows > 0) {
    b.sum = *sum;
    b.sum_blocks = row_sum_blocks(*sum, threads);
  }
  void (*kernel)(FftBatch<OPS>);
  long long blocks = tiles;
  if constexpr (N > 32) {
    kernel = plane_major ? coop_kernel<N, T, OPS, INVERSE, true>() : coop_kernel<N, T, OPS, INVERSE, false>();
    blocks = coop_grid(coop_shape(N, INVERSE, plane_major), tiles);
  } else {
    if (threads != block_threads<N, T>()) return cudaErrorInvalidConfiguration;
    kernel = line_kernel<N, T, OPS, INVERSE, kPlanes>();
    if constexpr (fft_modes_supported(N) && (OPS == 1 || !INVERSE))
      if (mode == kTiles) kernel = line_kernel<N, T, OPS, INVERSE, kTiles>();
    if constexpr (fft_modes_supported(N) && OPS == 1)
      if (mode == kReference) kernel = line_kernel<N, T, OPS, INVERSE, kReference>();
  }
  if (mode != kPlanes && !fft_modes_supported(N)) return cudaErrorInvalidConfiguration;
  if (mode == kTiles && INVERSE && OPS > 1) return cudaErrorInvalidConfiguration;  // no pass inverts two views at once
  if (mode == kReference && (OPS > 1 || ops[0].n_rows != 1 || ops[0].view.nw)) return cudaErrorInvalidConfiguration;
  cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
  if (e != cudaSuccess) return e;
  e = launch_dependent(kernel, dim3((unsigned)(blocks + b.sum_blocks)), threads, smem, stream, b);
  count_launch();
  return e;
}

// Sizes below 8 points are those of stand-alone transforms, one operand each.
template <int N, bool INVERSE>
cudaError_t run_ops(const FftParams* ops, int count, const RowSum* sum, cudaStream_t s) {
  if (count == 1) return run_batch<N, 1, INVERSE>(ops, count, sum, s);
  if constexpr (N >= 8)
    return run_batch<N, INVERSE ? kMaxInverseOps : kMaxFftOps, INVERSE>(ops, count, sum, s);
  else
    return cudaErrorInvalidValue;
}

template <bool INVERSE>
cudaError_t dispatch(const FftParams* ops, int count, const RowSum* sum, int N, cudaStream_t s) {
  if (count < 1 || count > (INVERSE ? kMaxInverseOps : kMaxFftOps)) return cudaErrorInvalidValue;
  for (int i = 0; i < count; ++i)
    if (ops[i].n_rows > 65535 || !spectrum_fits(ops[i], N)) return cudaErrorInvalidConfiguration;
  switch (N) {
    case 2: return run_ops<2, INVERSE>(ops, count, sum, s);
    case 4: return run_ops<4, INVERSE>(ops, count, sum, s);
    case 8: return run_ops<8, INVERSE>(ops, count, sum, s);
    case 16: return run_ops<16, INVERSE>(ops, count, sum, s);
    case 32: return run_ops<32, INVERSE>(ops, count, sum, s);
    case 64: return run_ops<64, INVERSE>(ops, count, sum, s);
    case 128: return run_ops<128, INVERSE>(ops, count, sum, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

int sm_count() {
  constexpr int kMaxDevices = 64;
  static std::atomic<int> cache[kMaxDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) dev = 0;
  int n = cache[dev].load(std::memory_order_relaxed);
  if (n > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) {
    cudaGetLastError();
    return 1;  // not cached: asked again at the next launch
  }
  cache[dev].store(n, std::memory_order_relaxed);
  return n;
}

void count_launch(int n) { g_launches.fetch_add(static_cast<uint64_t>(n), std::memory_order_relaxed); }
uint64_t launch_count() { return g_launches.load(std::memory_order_relaxed); }

cudaError_t launch_forward(const FftParams* ops, int count, int N, cudaStream_t stream) {
  return dispatch<false>(ops, count, nullptr, N, stream);
}

cudaError_t launch_inverse(const FftParams* ops, int count, const RowSum* sum, int N, cudaStream_t stream) {
  return dispatch<true>(ops, count, sum, N, stream);
}

namespace {

template <int N>
cudaError_t run_1d(bool inverse, const FftParams& p, cudaStream_t stream) {
  constexpr int T = fft_tile(N);
  const FftGeom g = inverse ? inverse_geom(N, T, p.h, p.w) : forward_geom(N, T, p.h, p.w, 0, p.off_x);
  void (*kernel)(FftParams, FftGeom) = inverse ? fft1d_inverse_kernel<N, T> : fft1d_forward_kernel<N, T>;
  cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), g.smem_bytes);
  if (e != cudaSuccess) return e;
  e = launch_dependent(kernel, dim3((p.n_inner + T - 1) / T), g.threads, g.smem_bytes, stream, p, g);
  count_launch();
  return e;
}

}  // namespace

// Rows [0, rows) of `n` floats each, transform size N: full blocks of N rows, then the rest.
cudaError_t launch_fft1d(bool inverse, const float* real_in, float* real_out, float2* spec, long long rows, int n,
                         int N, int offset, cudaStream_t stream) {
  if (N >= 64) return launch_fft1d_lines(inverse, real_in, real_out, spec, rows, n, N, offset, stream);
  const int KX = N / 2 + 1;
  for (int part = 0; part < 2; ++part) {
    const long long first = part == 0 ? 0 : rows / N * N;
    const int h = part == 0 ? N : (int)(rows % N);
    const long long planes = part == 0 ? rows / N : 1;
    if (h == 0 || planes == 0) continue;
    if (planes > 0x7fffffff) return cudaErrorInvalidValue;
    FftParams p{};
    p.real_in = real_in ? real_in + first * n : nullptr;
    p.real_out = real_out ? real_out + first * n : nullptr;
    p.spec = spec + first * KX;
    p.h = h;
    p.w = n;
    p.off_y = 0;
    p.off_x = offset;
    p.n_rows = 1;
    p.n_inner = (int)planes;
    p.kc = (int)planes;
    p.real_row_stride = 0;
    p.real_inner_stride = 1;
    cudaError_t e;
    switch (N) {
      case 2: e = run_1d<2>(inverse, p, stream); break;
      case 4: e = run_1d<4>(inverse, p, stream); break;
      case 8: e = run_1d<8>(inverse, p, stream); break;
      case 16: e = run_1d<16>(inverse, p, stream); break;
      case 32: e = run_1d<32>(inverse, p, stream); break;
      default: e = cudaErrorInvalidValue;
    }
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

namespace {

// The reference's 2-D frequency tensor (planes, N/2+1, N, 2) holds, for 8 <= N <= 32, rows ky <= N/2
// of the full spectrum, which the transforms store and load themselves (kReference), and for the other
// sizes the half spectrum along x stored transposed (element [kx][ky] = X[ky][kx], kx <= N/2)
// (test/test_FFTModule.lua:310-342), which the kernels below convert from and to the library's half
// spectrum [bin = ky*(N/2+1) + kx][plane].
__global__ void __launch_bounds__(256)
spectrum_to_reference_kernel(const float2* __restrict__ spec, float2* __restrict__ ref, long long planes, int kc,
                             int N) {
  grid_dependency_wait();
  const int KX = N / 2 + 1;
  const long long per_plane = (long long)KX * N;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < planes * per_plane;
       i += (long long)gridDim.x * blockDim.x) {
    const long long p = i / per_plane;
    const int r = (int)(i - p * per_plane);
    const int a = r / N, b = r - a * N;  // element [kx = a][ky = b]
    ref[i] = spec[((long long)b * KX + a) * kc + p];
  }
}

__global__ void __launch_bounds__(256)
reference_to_spectrum_kernel(const float2* __restrict__ ref, float2* __restrict__ spec, long long planes, int kc,
                             int N) {
  grid_dependency_wait();
  const int KX = N / 2 + 1;
  const long long bins = (long long)KX * N;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < bins * kc;
       i += (long long)gridDim.x * blockDim.x) {
    const long long bin = i / kc;
    const long long p = i - bin * kc;
    float2 v = make_float2(0.f, 0.f);  // the padding planes of the library's layout are zero
    if (p < planes) {
      const int ky = (int)(bin / KX), kx = (int)(bin - (long long)ky * KX);
      v = ref[p * bins + kx * N + ky];
    }
    spec[i] = v;
  }
}

}  // namespace

cudaError_t launch_spectrum_layout(bool to_reference, const float2* src, float2* dst, long long planes, int kc, int N,
                                   cudaStream_t stream) {
  const long long total = to_reference ? planes * (N / 2 + 1) * N : (long long)(N / 2 + 1) * N * kc;
  const long long want = (total + 255) / 256, cap = (long long)sm_count() * 16;
  const int blocks = (int)(want < 1 ? 1 : want < cap ? want : cap);
  const cudaError_t e = launch_dependent(to_reference ? spectrum_to_reference_kernel : reference_to_spectrum_kernel,
                                         dim3(blocks), 256, 0, stream, src, dst, planes, kc, N);
  count_launch();
  return e;
}

}  // namespace fbfft

