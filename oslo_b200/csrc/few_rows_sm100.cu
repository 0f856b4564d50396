// Products of a few rows (1 to 64) with a weight matrix: y[m, n] = act([x1 | x2][m, :] . W[:, n] + bias[n]) + res[m, n], with an
// optional LayerNorm of x1 in front. Decode steps are made of these; they are bound by how fast W streams out of HBM and, for small
// models, by launches.
//
// Up to 8 rows (few_rows_kernel): a warp owns a tile of 32 columns (64 for [K, N] weights) over a range of k, the block's other warps
// and the CTAs of a cluster own the other ranges, and the partial sums meet in shared memory (first of the block, then, pushed through
// distributed shared memory, of the cluster), so there is no workspace in global memory and no second kernel. Every lane fetches with
// cp.async the 16-byte pieces that it will feed to the tensor cores itself: which k a lane's fragment elements stand for is free as
// long as both operands agree, so a lane takes eight consecutive k of a row for two m16n8k16 steps and shared memory serves as a deep
// private queue, without barriers and without bank conflicts. mma.sync suffices there: with 8 rows the tensor cores idle either way.
// 9 to 64 rows (few_rows_tc_kernel): tcgen05.
// In chains of launches on weights that are in no cache (bf16): 1 row, [28672, 4096] 39 us, 6.05 TB/s; 8 rows, [14336, 2048] 11.8 us
// (split-k GEMM on 128-row tiles and the sum of its planes: 15.5 + 2.7); 32 rows, [28672, 4096] 43 us, [4096, 20480] 30 us (an average
// of 43 + 4.6 before); 1 row, [768, 3072]^T 4.0 us (4.9 + 3.1 before). A copy of the weights would take 36, 9.1, 36, 26 and 0.7 us.
//
// The launches are programmatic: a block asks for the first pieces of W in L2 (a hint: nothing is read) while the kernel before it
// still runs (11.8 us; 12.3 without), and reads W, x and the residual only after that kernel is complete.
//
// Reference behaviour covered: the linear layers of one iteration of the token loop of oslo/generation_utils.py:1269-1361.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "oslo_kernels.h"
#include "ptx.cuh"

namespace oslo {
int make_tma_2d_16bit(CUtensorMap* map, const void* ptr, uint64_t inner, uint64_t outer, uint64_t row_stride_elems, uint32_t box_rows,
                      bool fp16);   // gemm_sm100.cu
}

namespace oslo {

struct FewRows {
  const void* x1; const void* x2;          // [M, K1], [M, K2]
  const void* w[3];                        // [Np, K] each (KN: [K, N], one)
  const void* bias; const void* res;       // [N], [M, N]
  const void* ln_w; const void* ln_b;      // [K]
  void* out;
  long long sx, sw, so;                    // strides of stacked products (gridDim.y)
  float eps;
  int ld1, ld2, ldw, ldr, ldo, M, N, Np, K1, K, gelu_from, splits;
};

template <typename T> struct Few;
template <> struct Few<__nv_bfloat16> {
  static constexpr bool FP16 = false;
  static __device__ __forceinline__ float2 to2(uint32_t v) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v)); }
  static __device__ __forceinline__ float to(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ __nv_bfloat16 from(float v) { return __float2bfloat16_rn(v); }
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
  static __device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
};
template <> struct Few<__half> {
  static constexpr bool FP16 = true;
  static __device__ __forceinline__ float2 to2(uint32_t v) { return __half22float2(*reinterpret_cast<const __half2*>(&v)); }
  static __device__ __forceinline__ float to(__half v) { return __half2float(v); }
  static __device__ __forceinline__ __half from(float v) { return __float2half_rn(v); }
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    const __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
  static __device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
};

__device__ __forceinline__ float few_gelu(float x) {
  const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  return 0.5f * x * (1.0f + tanhf(u));
}
// 16 bytes, or zeros where `live` is false (the address must be valid either way). W goes past L1; x may be shared by a block's warps.
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp16_l1(uint32_t dst, const void* src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ uint4 lds16(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
  return v;
}

constexpr int FR_WARPS = 8;

// KN: W is [K, N] (a lane then holds 8 columns of 8 k, and the fragments are made with byte permutes); LN: LayerNorm of x1, which
// every block computes for itself and keeps in shared memory (at most FR_LN_ELEMS values).
constexpr int FR_ROWS = 8, FR_LN_ELEMS = 8192, FR_LN_PAD = 32;
template <bool KN, bool LN> struct FewShape {
  static constexpr int COLS = KN ? 64 : 32, ACC = COLS / 16;                 // columns of a block, tiles of 16 of them
  static constexpr int WSLOTS = KN ? 8 : 4, SLOTS = WSLOTS + (LN ? 0 : 1);
  static constexpr int STAGE = SLOTS * 512 * FR_WARPS;                       // bytes of one stage of all warps
  static constexpr int RED_LD = COLS + 4;                                    // row stride of the partial sums: rows 2t fall 8 banks apart
  static constexpr int RED = FR_WARPS * FR_ROWS * RED_LD * 4, INBOX = (FR_ROWS * COLS + 8) * 4;
  static constexpr int XS = LN ? (FR_LN_ELEMS + FR_ROWS * FR_LN_PAD) * 2 : 0;
  static constexpr int STAGES = (112 * 1024 - RED - INBOX - XS) / STAGE;     // two blocks fit an SM
  static constexpr int SMEM = STAGES * STAGE + RED + INBOX + XS;
  static_assert(STAGES >= 2, "shared memory of a block");
};

template <typename T, bool KN, bool LN>
__global__ void __launch_bounds__(FR_WARPS * 32, 2) few_rows_kernel(const FewRows p) {
  using S = FewShape<KN, LN>;
  constexpr int ACC = S::ACC, THREADS = FR_WARPS * 32;
  extern __shared__ __align__(16) unsigned char few_smem[];
  __shared__ float stat[2][8];                  // LayerNorm: mean and reciprocal deviation of each row
  __shared__ float part[2][FR_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int rank = blockIdx.x % p.splits, tile0 = blockIdx.x / p.splits, tile_step = gridDim.x / p.splits;   // clusters: `splits` blocks
  const int tiles = (p.N + S::COLS - 1) / S::COLS;
  const bool several = p.splits > 1;
  const T* x1 = reinterpret_cast<const T*>(p.x1) + blockIdx.y * p.sx;
  const T* x2 = reinterpret_cast<const T*>(p.x2);
  // the peers' shared memory may be written once they have started; this is waited for before the first write
  if (several) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  // this warp's range of 32-wide k steps, the same for every tile
  const int steps = (p.K + 31) / 32, ranges = p.splits * FR_WARPS, range = rank * FR_WARPS + warp;
  const int s0 = static_cast<int>(static_cast<long long>(steps) * range / ranges);
  const int s1 = static_cast<int>(static_cast<long long>(steps) * (range + 1) / ranges);
  // where this lane's pieces of W start (row n of its tile at k = 0; KN: row k = 0 at column n0 + 8 g)
  const T* wp[KN ? 1 : 4];
  bool wlive[KN ? 1 : 4];
  auto point = [&](int tile) {
    if constexpr (KN) {
      const int n = tile * S::COLS + 8 * g;
      wlive[0] = n < p.N;
      wp[0] = reinterpret_cast<const T*>(p.w[0]) + blockIdx.y * p.sw + (wlive[0] ? n : 0);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int n = tile * S::COLS + i * 8 + g;
        wlive[i] = n < p.N;
        const int nn = wlive[i] ? n : 0, which = nn / p.Np;
        wp[i] = reinterpret_cast<const T*>(which == 0 ? p.w[0] : (which == 1 ? p.w[1] : p.w[2])) + blockIdx.y * p.sw +
                static_cast<long long>(nn - which * p.Np) * p.ldw;
      }
    }
  };
  point(tile0);
  if constexpr (KN) {
    if (wlive[0] && (g & 3) == 0)
      for (int k = s0 * 32 + t; k < min(p.K, min(s1, s0 + 4) * 32); k += 4) asm volatile("prefetch.global.L2 [%0];" ::"l"(wp[0] + static_cast<long long>(k) * p.ldw));
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (wlive[i])
        for (int k = s0 * 32 + t * 64; k < min(p.K, min(s1, s0 + 4) * 32); k += 256) asm volatile("prefetch.global.L2 [%0];" ::"l"(wp[i] + k));
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");

  // the ring runs on through the tiles: the next one's pieces are on their way while this one's sums meet
  const uint32_t ring = smem_u32(few_smem) + (warp * S::SLOTS * 32 + lane) * 16;
  int ftile = tile0, fstep = s0, fslot = 0;
  auto fetch = [&]() {
    if (ftile < tiles && s0 < s1) {
      const uint32_t at = ring + fslot * S::STAGE;
      const int k = fstep * 32 + 8 * t;
      const bool in = k < p.K;                  // K % 8 == 0: a piece is inside or outside
      const int kk = in ? k : 0;
      if constexpr (KN) {
#pragma unroll
        for (int i = 0; i < 8; ++i) cp16(at + i * 512, wp[0] + static_cast<long long>(kk + i) * p.ldw, in && wlive[0]);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) cp16(at + i * 512, wp[i] + kk, in && wlive[i]);
      }
      if constexpr (!LN) {
        const bool second = kk >= p.K1;
        const T* xb = second ? x2 + (kk - p.K1) : x1 + kk;
        const long long ld = second ? p.ld2 : p.ld1;
        cp16_l1(at + S::WSLOTS * 512, xb + (g < p.M ? g * ld : 0), in && g < p.M);
      }
      if (++fslot == S::STAGES) fslot = 0;
      if (++fstep == s1) {
        fstep = s0;
        ftile += tile_step;
        point(ftile);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < S::STAGES - 1; ++i) fetch();

  const int xs_ld = p.K + FR_LN_PAD;            // 64 bytes of padding: the rows' pieces fall into different banks
  T* xs = reinterpret_cast<T*>(few_smem + S::STAGES * S::STAGE + S::RED + S::INBOX);
  if constexpr (LN) {                           // statistics of the rows: 8, 4, 2 or 1 warps to a row, twice over x (the second from L1)
    const int wpr = p.M > 4 ? 1 : (p.M > 2 ? 2 : (p.M > 1 ? 4 : 8));
    const int row = warp / wpr, li = (warp % wpr) * 32 + lane;
    const bool live = row < p.M;
    const T* xr = x1 + static_cast<long long>(live ? row : 0) * p.ld1;
    float mean = 0.f;
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
      float s = 0.f;
      for (int c = li * 8; c < p.K; c += wpr * 256) {
        const uint4 v = *reinterpret_cast<const uint4*>(xr + c);
        const uint32_t q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = Few<T>::to2(q[j]);
          s += pass == 0 ? f.x + f.y : (f.x - mean) * (f.x - mean) + (f.y - mean) * (f.y - mean);
        }
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
      if (lane == 0) part[pass][warp] = s;
      __syncthreads();
      float tot = 0.f;
      for (int i = 0; i < wpr; ++i) tot += part[pass][row * wpr + i];
      if (pass == 0) mean = tot / p.K;
      else if (live && li == 0) { stat[0][row] = mean; stat[1][row] = rsqrtf(tot / p.K + p.eps); }
    }
    __syncthreads();
    for (int e = threadIdx.x * 8; e < p.M * p.K; e += THREADS * 8) {       // rounded to T, as the LayerNorm kernel stores it
      const int m = e / p.K, k = e - m * p.K;
      const float mu = stat[0][m], rs = stat[1][m];
      const uint4 v = *reinterpret_cast<const uint4*>(x1 + static_cast<long long>(m) * p.ld1 + k);
      const uint4 gw = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.ln_w) + k);
      const uint4 gb = p.ln_b ? *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.ln_b) + k) : make_uint4(0, 0, 0, 0);
      const uint32_t q[4] = {v.x, v.y, v.z, v.w}, a[4] = {gw.x, gw.y, gw.z, gw.w}, b[4] = {gb.x, gb.y, gb.z, gb.w};
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = Few<T>::to2(q[j]), w2 = Few<T>::to2(a[j]), b2 = Few<T>::to2(b[j]);
        o[j] = Few<T>::pack((f.x - mu) * rs * w2.x + b2.x, (f.y - mu) * rs * w2.y + b2.y);
      }
      *reinterpret_cast<uint4*>(xs + m * xs_ld + k) = make_uint4(o[0], o[1], o[2], o[3]);
    }
    __syncthreads();
  }

  float* red = reinterpret_cast<float*>(few_smem + S::STAGES * S::STAGE);
  float* inbox = red + S::RED / 4;              // [splits][share of the tile's elements]
  const int elems = p.M * S::COLS, share = (elems + p.splits - 1) / p.splits;
  T* out = reinterpret_cast<T*>(p.out) + blockIdx.y * p.so;
  int slot = 0;
  bool met = !several;
  for (int tile = tile0; tile < tiles; tile += tile_step) {
    float acc[ACC][4];
#pragma unroll
    for (int r = 0; r < ACC; ++r)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[r][i] = 0.f;
    for (int step = s0; step < s1; ++step) {
      fetch();                                  // into the slot that the step before this one has read
      asm volatile("cp.async.wait_group %0;" ::"n"(S::STAGES - 1) : "memory");
      const uint32_t at = ring + slot * S::STAGE;
      if (++slot == S::STAGES) slot = 0;
      uint4 xv;
      if constexpr (LN) {
        const int k = step * 32 + 8 * t;
        xv = g < p.M && k < p.K ? lds16(smem_u32(xs + g * xs_ld + k)) : make_uint4(0, 0, 0, 0);
      } else {
        xv = lds16(at + S::WSLOTS * 512);
      }
      if constexpr (KN) {
        uint4 wv[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) wv[i] = lds16(at + i * 512);
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            auto word = [r](const uint4& v) { return r == 0 ? v.x : (r == 1 ? v.y : (r == 2 ? v.z : v.w)); };
            const uint32_t u0 = word(wv[4 * j]), u1 = word(wv[4 * j + 1]), u2 = word(wv[4 * j + 2]), u3 = word(wv[4 * j + 3]);
            const uint32_t a0 = __byte_perm(u0, u1, 0x5410), a1 = __byte_perm(u0, u1, 0x7632);
            const uint32_t a2 = __byte_perm(u2, u3, 0x5410), a3 = __byte_perm(u2, u3, 0x7632);
            Few<T>::mma(acc[r], a0, a1, a2, a3, j ? xv.z : xv.x, j ? xv.w : xv.y);
          }
      } else {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const uint4 u = lds16(at + (2 * r) * 512), v = lds16(at + (2 * r + 1) * 512);
          Few<T>::mma(acc[r], u.x, v.x, u.y, v.y, xv.x, xv.y);
          Few<T>::mma(acc[r], u.z, v.z, u.w, v.w, xv.z, xv.w);
        }
      }
    }
    // partial sums: of the block's warps in shared memory, then every element's from the cluster's blocks in its owner's inbox
    __syncthreads();                            // the sums of the tile before this one are read
#pragma unroll
    for (int r = 0; r < ACC; ++r)
      for (int i = 0; i < 4; ++i) {
        const int n = KN ? 8 * g + 2 * r + (i >> 1) : r * 16 + g + (i >> 1) * 8;
        red[(warp * FR_ROWS + 2 * t + (i & 1)) * S::RED_LD + n] = acc[r][i];
      }
    __syncthreads();
    auto finish = [&](int m, int c, float v) {
      const int n = tile * S::COLS + c;
      if (n >= p.N) return;
      if (p.bias) v += Few<T>::to(reinterpret_cast<const T*>(p.bias)[n]);
      if (p.gelu_from >= 0 && n >= p.gelu_from) v = few_gelu(v);
      if (p.gelu_from == OSLO_ACT_RELU2) { v = fmaxf(v, 0.f); v *= v; }
      if (p.res) v += Few<T>::to(reinterpret_cast<const T*>(p.res)[static_cast<long long>(m) * p.ldr + n]);
      out[static_cast<long long>(m) * p.ldo + n] = Few<T>::from(v);
    };
    if (!met) {
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
      met = true;
    }
    for (int e = threadIdx.x; e < elems; e += THREADS) {
      const int m = e / S::COLS, c = e % S::COLS;
      float v = 0.f;
#pragma unroll
      for (int i = 0; i < FR_WARPS; ++i) v += red[(i * FR_ROWS + m) * S::RED_LD + c];
      if (several) {
        const int owner = e / share;
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(map_to_cta(smem_u32(inbox + rank * share + (e - owner * share)), owner)), "f"(v) : "memory");
      } else {
        finish(m, c, v);
      }
    }
    if (several) {                              // only shapes of one tile per cluster are split (few_launch): the inbox is used once
      cluster_sync_all();
      for (int e = threadIdx.x; e < share && rank * share + e < elems; e += THREADS) {
        float v = 0.f;
        for (int r = 0; r < p.splits; ++r) v += inbox[r * share + e];
        finish((rank * share + e) / S::COLS, (rank * share + e) % S::COLS, v);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// One row and [N, K] weights: four columns per block of 256 threads over the whole range of k, in 32-bit FMAs, with 2 x 4 weight loads of
// 16 bytes per lane on their way. No sums meet but a block's, which is what few outputs gain from, and weights of 64 M values and more
// stream faster (one_row_better has the line).
constexpr int OR_THREADS = 256, OR_COLS = 4;
__device__ __forceinline__ uint4 ld_stream_16(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
template <typename T>
__device__ __forceinline__ void one_row_segment(const T* __restrict__ x, int K, const T* __restrict__ w, int ldw, float (&acc)[OR_COLS]) {
  constexpr int STEP = OR_THREADS * 8;
  for (int k = threadIdx.x * 8; k < K; k += 2 * STEP) {
    const bool second = k + STEP < K;
    uint4 wv[2][OR_COLS];
#pragma unroll
    for (int c = 0; c < OR_COLS; ++c) {
      wv[0][c] = ld_stream_16(w + static_cast<size_t>(c) * ldw + k);
      wv[1][c] = second ? ld_stream_16(w + static_cast<size_t>(c) * ldw + k + STEP) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (u == 1 && !second) break;
      const uint4 xv = *reinterpret_cast<const uint4*>(x + k + u * STEP);
      const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
      for (int c = 0; c < OR_COLS; ++c) {
        const uint32_t ww[4] = {wv[u][c].x, wv[u][c].y, wv[u][c].z, wv[u][c].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 a = Few<T>::to2(xw[j]), b = Few<T>::to2(ww[j]);
          acc[c] = fmaf(a.x, b.x, acc[c]);
          acc[c] = fmaf(a.y, b.y, acc[c]);
        }
      }
    }
  }
}
template <typename T>
__global__ void __launch_bounds__(OR_THREADS) one_row_kernel(const FewRows p) {
  __shared__ float red[OR_THREADS / 32][OR_COLS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const T* x1 = reinterpret_cast<const T*>(p.x1) + blockIdx.y * p.sx;
  const T* W = reinterpret_cast<const T*>(p.w[0]) + blockIdx.y * p.sw;
  T* out = reinterpret_cast<T*>(p.out) + blockIdx.y * p.so;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // the next kernel's blocks only where these leave room: blocks that walk several groups of columns fill the SMs to the end
  if (p.N <= OR_COLS * gridDim.x) asm volatile("griddepcontrol.launch_dependents;");
  for (int n0 = blockIdx.x * OR_COLS; n0 < p.N; n0 += gridDim.x * OR_COLS) {     // N % OR_COLS == 0
    float acc[OR_COLS] = {0.f, 0.f, 0.f, 0.f};
    const T* w = W + static_cast<size_t>(n0) * p.ldw;
    one_row_segment<T>(x1, p.K1, w, p.ldw, acc);
    if (p.x2 != nullptr) one_row_segment<T>(reinterpret_cast<const T*>(p.x2), p.K - p.K1, w + p.K1, p.ldw, acc);
#pragma unroll
    for (int c = 0; c < OR_COLS; ++c) {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], off);
      if (lane == 0) red[warp][c] = acc[c];
    }
    __syncthreads();
    if (threadIdx.x < OR_COLS) {
      const int n = n0 + threadIdx.x;
      float v = 0.f;
#pragma unroll
      for (int i = 0; i < OR_THREADS / 32; ++i) v += red[i][threadIdx.x];
      if (p.bias) v += Few<T>::to(reinterpret_cast<const T*>(p.bias)[n]);
      if (p.gelu_from >= 0 && n >= p.gelu_from) v = few_gelu(v);
      if (p.gelu_from == OSLO_ACT_RELU2) { v = fmaxf(v, 0.f); v *= v; }
      if (p.res) v += Few<T>::to(reinterpret_cast<const T*>(p.res)[n]);
      out[n] = Few<T>::from(v);
    }
    __syncthreads();
  }
}
// Columns of all products that one wave of blocks covers, or weights large enough to be bound by bandwidth alone (bf16, cold weights, us,
// one_row_kernel and few_rows_kernel: [768, 768] 2.4 and 2.9, [2304, 768] 3.0 and 3.5, [2048, 8192] 7.7 and 7.9, [4096, 20480] 28.2 and 31.9,
// [50400, 4096] 63.5 and 69.6; in between [3072, 768] 4.4 and 3.7, [4096, 4096] 8.7 and 7.9, [8192, 2048] 9.1 and 7.1)
static bool one_row_better(const FewRows& p, int stacked, int num_sms) {
  const long long cols = static_cast<long long>(p.N) * stacked;
  return p.M == 1 && p.N % OR_COLS == 0 && (cols <= 4ll * OR_COLS * num_sms || cols * p.K >= 64ll << 20);
}
template <typename T>
static int one_row_launch(const FewRows& p, int stacked, int num_sms, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(std::max(1, std::min(p.N / OR_COLS, 8 * num_sms / stacked))), stacked);
  cfg.blockDim = dim3(OR_THREADS);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, one_row_kernel<T>, p));
}

template <typename T, bool KN, bool LN>
static int few_launch(FewRows& p, int stacked, int num_sms, cudaStream_t st) {
  using S = FewShape<KN, LN>;
  auto kernel = few_rows_kernel<T, KN, LN>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM);
  if (e != cudaSuccess) return static_cast<int>(e);
  // two blocks per SM in one wave: k is cut over a cluster while that leaves room and every warp a step of its own, and more tiles
  // than blocks are walked
  const int tiles = (p.N + S::COLS - 1) / S::COLS, steps = (p.K + 31) / 32, room = std::max(1, 2 * num_sms / stacked);
  int splits = 1;
  while (splits < 8 && tiles * splits * 2 <= room && steps >= 2 * splits * FR_WARPS) splits *= 2;
  p.splits = splits;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(splits > 1 ? tiles * splits : std::min(tiles, room)), stacked);
  cfg.blockDim = dim3(FR_WARPS * 32);
  cfg.dynamicSmemBytes = S::SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = splits; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kernel, static_cast<const FewRows>(p)));
}

template <typename T>
static int few_dispatch(FewRows& p, bool kn, int parts, int num_sms, cudaStream_t st) {
  const bool ln = p.ln_w != nullptr;
  if (!kn && !ln && p.Np == p.N && one_row_better(p, parts, num_sms)) return one_row_launch<T>(p, parts, num_sms, st);
  if (kn) return ln ? few_launch<T, true, true>(p, parts, num_sms, st) : few_launch<T, true, false>(p, parts, num_sms, st);
  return ln ? few_launch<T, false, true>(p, parts, num_sms, st) : few_launch<T, false, false>(p, parts, num_sms, st);
}

// The same product for more than FR_ROWS rows on tcgen05: above, every warp fetches the fragments of x again. W is the
// 128-row operand here too and x the narrow one (MP = 16, 32 or 64 rows), so nothing is padded to a 128-row tile; one tile of 128
// columns and one range of k per CTA, the CTAs of a cluster share a tile's k range and add up through distributed shared memory.
// Warp 0 feeds the ring with TMA, warp 1 issues the MMAs, warps 2 to 5 read the accumulator.
struct FewTc {
  FewRows p;
  int* err;
  int stages;
};
constexpr int FT_THREADS = 192, FT_BN = 128, FT_BK = 64, FT_LD = FT_BN + 4, FT_EPI = 4;

template <typename T, int MP, bool KN>
__global__ void __launch_bounds__(FT_THREADS, 1) few_rows_tc_kernel(const __grid_constant__ CUtensorMap tw0, const __grid_constant__ CUtensorMap tw1,
                                                                    const __grid_constant__ CUtensorMap tw2, const __grid_constant__ CUtensorMap tx1,
                                                                    const __grid_constant__ CUtensorMap tx2, const FewTc a) {
  constexpr uint32_t W_BYTES = FT_BN * FT_BK * 2, STAGE = W_BYTES + MP * FT_BK * 2, TMEM_COLS = MP < 32 ? 32 : MP;
  extern __shared__ uint8_t few_tc_raw[];
  __shared__ uint64_t bars[2 * 16 + 1];         // full, empty, accumulator
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  const FewRows& p = a.p;
  const uint32_t ring = (smem_u32(few_tc_raw) + 1023u) & ~1023u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x % p.splits, tile = blockIdx.x / p.splits;
  const int kblocks = (p.K + FT_BK - 1) / FT_BK;
  const int kb0 = static_cast<int>(static_cast<long long>(kblocks) * rank / p.splits);
  const int kb1 = static_cast<int>(static_cast<long long>(kblocks) * (rank + 1) / p.splits);
  auto full = [&](int s) { return smem_u32(&bars[s]); };
  auto empty = [&](int s) { return smem_u32(&bars[16 + s]); };
  const uint32_t done = smem_u32(&bars[32]);
  if (threadIdx.x == 0) {
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    mbar_init(done, 1);
    abort_word = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_slot), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t acc = tmem_slot;
  const int n_tile = tile * FT_BN, which = n_tile / p.Np, n0 = n_tile - which * p.Np;
  const CUtensorMap* tw = which == 0 ? &tw0 : (which == 1 ? &tw1 : &tw2);
  if (threadIdx.x == 0) {
    tma_prefetch_desc(tw);
    tma_prefetch_desc(&tx1);
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(empty(stage), phase ^ 1, abort_flag, a.err, ERR_WAIT_EMPTY)) break;
        const uint32_t sw = ring + stage * STAGE;
        const int k0 = kb * FT_BK;
        mbar_expect_tx(full(stage), STAGE);
        if constexpr (KN) {                       // boxes {64 n, 64 k rows}
          tma_load_2d(sw, tw, full(stage), n0, k0);
          tma_load_2d(sw + 8192, tw, full(stage), n0 + 64, k0);
        } else {
          tma_load_2d(sw, tw, full(stage), k0, n0);
        }
        if (k0 < p.K1) tma_load_2d(sw + W_BYTES, &tx1, full(stage), k0, 0);
        else tma_load_2d(sw + W_BYTES, &tx2, full(stage), k0 - p.K1, 0);
        if (++stage == a.stages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = make_idesc_f16(FT_BN, MP, Few<T>::FP16 ? 0 : 1, KN ? 1 : 0, 0);
      constexpr uint32_t LBO = KN ? 8192u : 16u, STEP = KN ? 2048u : 32u;
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        ok = mbar_wait(full(stage), phase, abort_flag, a.err, ERR_WAIT_FULL);
        if (!ok) break;
        tc_fence_after();
        const uint32_t sw = ring + stage * STAGE;
#pragma unroll
        for (int k = 0; k < FT_BK / 16; ++k)
          umma_f16(acc, make_smem_desc(sw + k * STEP, LBO, 1024), make_smem_desc(sw + W_BYTES + k * 32, 16, 1024), idesc, kb != kb0 || k != 0);
        umma_commit(empty(stage));
        if (++stage == a.stages) { stage = 0; phase ^= 1; }
      }
      if (ok) umma_commit(done);
    }
  }
  __syncwarp();
  // column of the tile = TMEM lane; the ring is free once the last MMA has read it
  float* red = reinterpret_cast<float*>(few_tc_raw + (ring - smem_u32(few_tc_raw)));
  if (warp >= 2) {
    const int quad = warp & 3;
    if (mbar_wait_warp(done, 0, abort_flag, a.err, ERR_WAIT_TMEM_FULL)) {
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < MP; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32(acc + (static_cast<uint32_t>(quad * 32) << 16) + c, r);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (c + i < MP && c + i < p.M) red[(c + i) * FT_LD + quad * 32 + lane] = __uint_as_float(r[i]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {                              // give copies that are still in flight time to land
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) {
    }
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(acc, TMEM_COLS);
  }
  if (p.splits > 1) cluster_sync_all();
  T* out = reinterpret_cast<T*>(p.out);
  const uint32_t base = smem_u32(red);
  auto finish = [&](int m, int n, float v) {
    if (p.bias) v += Few<T>::to(reinterpret_cast<const T*>(p.bias)[n]);
    if (p.gelu_from >= 0 && n >= p.gelu_from) v = few_gelu(v);
    if (p.gelu_from == OSLO_ACT_RELU2) { v = fmaxf(v, 0.f); v *= v; }
    if (p.res) v += Few<T>::to(reinterpret_cast<const T*>(p.res)[static_cast<long long>(m) * p.ldr + n]);
    out[static_cast<long long>(m) * p.ldo + n] = Few<T>::from(v);
  };
  if (p.splits == 1) {
#pragma unroll 1
    for (int e = threadIdx.x; e < p.M * FT_BN; e += FT_THREADS)
      if (n_tile + e % FT_BN < p.N) finish(e / FT_BN, n_tile + e % FT_BN, red[e / FT_BN * FT_LD + e % FT_BN]);
    return;
  }
  // FT_EPI elements of a thread at a time, all their parts on the way before the first is added: one by one, 64 rows waited for their
  // peers' memory eleven times over (64 rows, [1024, 640]: 8.5 us, 7.9 so)
  const int step = FT_THREADS * p.splits;
#pragma unroll 1
  for (int e0 = threadIdx.x + rank * FT_THREADS; e0 < p.M * FT_BN; e0 += FT_EPI * step) {
    float f[FT_EPI][8];
#pragma unroll
    for (int u = 0; u < FT_EPI; ++u) {
      const int e = e0 + u * step, m = e / FT_BN, c = e % FT_BN;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        f[u][r] = 0.f;
        if (e < p.M * FT_BN && r < p.splits)
          asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(f[u][r]) : "r"(map_to_cta(base + (m * FT_LD + c) * 4, r)) : "memory");
      }
    }
    float v[FT_EPI];
#pragma unroll
    for (int u = 0; u < FT_EPI; ++u) {
      v[u] = 0.f;
#pragma unroll
      for (int r = 0; r < 8; ++r) v[u] += f[u][r];
    }
#pragma unroll 1
    for (int u = 0; u < FT_EPI; ++u) {            // not unrolled: the epilogue's code is fetched anew by every launch
      const int e = e0 + u * step, n = n_tile + e % FT_BN;
      if (e < p.M * FT_BN && n < p.N) finish(e / FT_BN, n, u == 0 ? v[0] : (u == 1 ? v[1] : (u == 2 ? v[2] : v[3])));
    }
  }
  cluster_sync_all();                             // no block leaves while another may still read its sums
}

template <typename T, int MP, bool KN>
static int few_tc_launch(const FewRows& p0, int parts, int* err, int num_sms, cudaStream_t st) {
  constexpr int STAGE = FT_BN * FT_BK * 2 + MP * FT_BK * 2;
  auto kernel = few_rows_tc_kernel<T, MP, KN>;     // a runtime call first: the tensor-map encoder needs the context on this thread
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024);
  if (e != cudaSuccess) return static_cast<int>(e);
  FewTc a = {};
  a.p = p0; a.err = err;
  FewRows& p = a.p;
  // about two CTAs per SM, in one wave
  const int tiles = (p.N + FT_BN - 1) / FT_BN, kblocks = (p.K + FT_BK - 1) / FT_BK;
  int splits = 1;
  while (splits < 8 && tiles * splits * 2 <= 2 * num_sms && kblocks >= 4 * splits) splits *= 2;
  p.splits = splits;
  a.stages = 110 * 1024 / STAGE;                  // two CTAs fit an SM (one with all of its memory: clusters of eight find no room)
  const int smem = std::max(a.stages * STAGE, MP * FT_LD * 4) + 1024;
  CUtensorMap tw[3], tx[2];
  const bool fp16 = Few<T>::FP16;
  for (int i = 0; i < 3; ++i) {
    const void* w = p.w[i < parts ? i : 0];
    const int rc = KN ? make_tma_2d_16bit(&tw[i], w, p.N, p.K, p.ldw, 64, fp16) : make_tma_2d_16bit(&tw[i], w, p.K, p.Np, p.ldw, FT_BN, fp16);
    if (rc) return rc;
  }
  int rc = make_tma_2d_16bit(&tx[0], p.x1, p.K1, p.M, p.ld1, MP, fp16);
  if (!rc) rc = p.x2 ? make_tma_2d_16bit(&tx[1], p.x2, p.K - p.K1, p.M, p.ld2, MP, fp16) : 0;
  if (rc) return rc - 1000;
  if (!p.x2) tx[1] = tx[0];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(tiles) * splits);
  cfg.blockDim = dim3(FT_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = splits; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kernel, tw[0], tw[1], tw[2], tx[0], tx[1], static_cast<const FewTc>(a)));
}

template <typename T>
static int few_tc_dispatch(const FewRows& p, bool kn, int parts, int* err, int num_sms, cudaStream_t st) {
  if (kn) {
    if (p.M <= 16) return few_tc_launch<T, 16, true>(p, parts, err, num_sms, st);
    if (p.M <= 32) return few_tc_launch<T, 32, true>(p, parts, err, num_sms, st);
    return few_tc_launch<T, 64, true>(p, parts, err, num_sms, st);
  }
  if (p.M <= 16) return few_tc_launch<T, 16, false>(p, parts, err, num_sms, st);
  if (p.M <= 32) return few_tc_launch<T, 32, false>(p, parts, err, num_sms, st);
  return few_tc_launch<T, 64, false>(p, parts, err, num_sms, st);
}

static bool off16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; }

}  // namespace oslo

extern "C" int oslo_few_rows(const void* x1, int ld1, int K1, const void* x2, int ld2, int K2, const void* w0, const void* w1,
                             const void* w2, int parts, int ldw, int w_kn, const void* bias, const void* res, int ldr,
                             const void* ln_w, const void* ln_b, float eps, void* out, int ldo, int M, int N, int gelu_from,
                             int dtype, int* err_word, int num_sms, cudaStream_t stream) {
  using namespace oslo;
  if (M <= 0 || N <= 0) return 0;
  if (x2 == nullptr) K2 = 0;
  if (M > 64 || K1 <= 0 || K1 % 8 || K2 % 8 || ld1 % 8 || ldw % 8 || (x2 && ld2 % 8) || parts < 1 || parts > 3 || N % parts) return -1;
  if (w_kn && (N % 8 || parts != 1)) return -1;
  if (ln_w && (M > FR_ROWS || x2 || static_cast<long long>(M) * K1 > FR_LN_ELEMS)) return -1;
  // above FR_ROWS rows: a k block of 64 comes from one of the inputs, a tile of 128 columns from one of the weights
  if (M > FR_ROWS && ((x2 && K1 % FT_BK) || (parts > 1 && (N / parts) % FT_BN))) return -1;
  const void* ptrs[7] = {x1, x2, w0, parts > 1 ? w1 : nullptr, parts > 2 ? w2 : nullptr, ln_w, ln_b};
  for (const void* p : ptrs)
    if (off16(p)) return -4;
  FewRows p = {};
  p.x1 = x1; p.x2 = x2; p.w[0] = w0; p.w[1] = parts > 1 ? w1 : w0; p.w[2] = parts > 2 ? w2 : w0;
  p.bias = bias; p.res = res; p.ln_w = ln_w; p.ln_b = ln_b; p.out = out; p.eps = eps;
  p.ld1 = ld1; p.ld2 = ld2; p.ldw = ldw; p.ldr = ldr; p.ldo = ldo; p.M = M; p.N = N; p.Np = N / parts;
  p.K1 = K1; p.K = K1 + K2; p.gelu_from = gelu_from;
  // [K, N] weights of more than 6 M values stream through the tensor cores whatever the rows: few_rows_kernel's transposed fragments hold
  // them at 3 TB/s ([4096, 28672], 1 and 8 rows: 77.8 and 79.9 us, 41.0 and 42.0 so; [768, 3072]: 4.3 and 4.8, 5.6)
  const bool kn = w_kn != 0;
  const bool tc = M > FR_ROWS || (kn && !ln_w && static_cast<long long>(p.K) * N > 6ll << 20 && (!x2 || K1 % FT_BK == 0));
  if (dtype == OSLO_DT_BF16)
    return tc ? few_tc_dispatch<__nv_bfloat16>(p, kn, parts, err_word, num_sms, stream) : few_dispatch<__nv_bfloat16>(p, kn, 1, num_sms, stream);
  if (dtype == OSLO_DT_FP16)
    return tc ? few_tc_dispatch<__half>(p, kn, parts, err_word, num_sms, stream) : few_dispatch<__half>(p, kn, 1, num_sms, stream);
  return -2;
}

// P products at once: x [P, M, K] and W [P, N, K] (strides sx, sw between them) -> out [P, M, N], M <= 8
extern "C" int oslo_few_rows_stacked(const void* x, int ldx, long long sx, const void* W, int ldw, long long sw, void* out, int P,
                                     int M, int N, int K, int dtype, int num_sms, cudaStream_t stream) {
  using namespace oslo;
  if (P <= 0 || M <= 0 || N <= 0) return 0;
  if (M > FR_ROWS || P > 65535 || K <= 0 || K % 8 || ldx % 8 || ldw % 8 || sx % 8 || sw % 8) return -1;
  if (off16(x) || off16(W)) return -4;
  FewRows p = {};
  p.x1 = x; p.w[0] = p.w[1] = p.w[2] = W; p.out = out;
  p.sx = sx; p.sw = sw; p.so = static_cast<long long>(M) * N;
  p.ld1 = ldx; p.ldw = ldw; p.ldo = N; p.M = M; p.N = N; p.Np = N; p.K1 = p.K = K; p.gelu_from = -1;
  if (dtype == OSLO_DT_BF16) return few_dispatch<__nv_bfloat16>(p, false, P, num_sms, stream);
  if (dtype == OSLO_DT_FP16) return few_dispatch<__half>(p, false, P, num_sms, stream);
  return -2;
}
