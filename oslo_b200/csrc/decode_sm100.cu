// Kernels of the single-token decode step: bound by how fast the KV cache streams out of HBM and by launch count, not by math. The
// weight products are in few_rows_sm100.cu.
//   * rotary_append_kernel: GPT-J rotary on q and k of the new token, q to a contiguous buffer, k and v written
//     into the static cache at the position held in device memory.
//   * prompt_append_kernel: the keys and values of a prompt into the cache.
//   * decode_attn_kernel: attention of one query per row over the cache, with the rotary and the append of the new token inside
//     when it is given one.
//
// Reference behaviour covered: one iteration of the token loop of oslo/generation_utils.py:1269-1361 through a
// GPT-J block (oslo/models/gptj/modeling_gptj.py:196-320: rotary at the cache offset, torch.cat cache growth,
// attention, out_proj, MLP, parallel residual).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math_constants.h>

#include "oslo_kernels.h"
#include "ptx.cuh"

namespace oslo {

template <typename T> struct DCvt;
template <> struct DCvt<__nv_bfloat16> {
  static __device__ __forceinline__ float2 to2(uint32_t v) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v)); }
  static __device__ __forceinline__ __nv_bfloat16 from(float v) { return __float2bfloat16_rn(v); }
  static __device__ __forceinline__ float to(__nv_bfloat16 v) { return __bfloat162float(v); }
};
template <> struct DCvt<__half> {
  static __device__ __forceinline__ float2 to2(uint32_t v) { return __half22float2(*reinterpret_cast<const __half2*>(&v)); }
  static __device__ __forceinline__ __half from(float v) { return __float2half_rn(v); }
  static __device__ __forceinline__ float to(__half v) { return __half2float(v); }
};

// One block per (batch row, head): rotary (pairs (2i, 2i+1) of the first rotary_dim dims, position pos[b]) on q and
// k; q -> q_out [B, H, D]; k, v -> cache[b, h, write_index[0], :]. q/k/v rows are [H * D] slices with row strides.
template <typename T>
__global__ void rotary_append_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v,
                                     long long ldq, long long ldk, long long ldv, T* __restrict__ q_out,
                                     T* __restrict__ kc, T* __restrict__ vc, const int* __restrict__ lengths,
                                     const long long* __restrict__ write_index, int H, int D, int Tmax, int rotary_dim,
                                     float log2_base, int* err) {
  const int b = blockIdx.y, h = blockIdx.x;
  const long long wi = write_index[0];
  if (wi < 0 || wi >= Tmax) {   // never write outside the cache
    OSLO_REPORT_BOUNDS(err);
    return;
  }
  const float pos = static_cast<float>(lengths[b]);
  const T* qp = q + b * ldq + static_cast<long long>(h) * D;
  const T* kp = k + b * ldk + static_cast<long long>(h) * D;
  const T* vp = v + b * ldv + static_cast<long long>(h) * D;
  T* qo = q_out + (static_cast<long long>(b) * H + h) * D;
  T* ko = kc + ((static_cast<long long>(b) * H + h) * Tmax + wi) * D;
  T* vo = vc + ((static_cast<long long>(b) * H + h) * Tmax + wi) * D;
  for (int i = threadIdx.x; i < D / 2; i += blockDim.x) {
    const int d0 = 2 * i;
    float q0 = DCvt<T>::to(qp[d0]), q1 = DCvt<T>::to(qp[d0 + 1]);
    float k0 = DCvt<T>::to(kp[d0]), k1 = DCvt<T>::to(kp[d0 + 1]);
    if (d0 < rotary_dim) {
      const float inv_freq = exp2f(-log2_base * (2.0f * i) / rotary_dim);   // same expression as rotary_kernel
      float sn, cs;
      sincosf(pos * inv_freq, &sn, &cs);
      const float a = q0 * cs - q1 * sn, bq = q1 * cs + q0 * sn;
      q0 = a; q1 = bq;
      const float c = k0 * cs - k1 * sn, dk = k1 * cs + k0 * sn;
      k0 = c; k1 = dk;
    }
    qo[d0] = DCvt<T>::from(q0); qo[d0 + 1] = DCvt<T>::from(q1);
    ko[d0] = DCvt<T>::from(k0); ko[d0 + 1] = DCvt<T>::from(k1);
    vo[d0] = vp[d0]; vo[d0 + 1] = vp[d0 + 1];
  }
}

// k, v [B, H, S, D] by strides -> cache[b, h, start + s, :], in 16-byte pieces, four in flight per thread. Bound by memory: the library's
// strided copies moved 134 MB in 108 us each (4 x 16 x 2048 x 256, one tensor).
template <typename V>
__global__ void __launch_bounds__(256) prompt_append_kernel(const V* __restrict__ k, const V* __restrict__ v, V* __restrict__ kc, V* __restrict__ vc,
                                                            long long k_sb, long long k_sh, long long k_ss, long long v_sb, long long v_sh,
                                                            long long v_ss, int H, int S, int per, int T, int start, long long total) {
  const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
  const V* src = blockIdx.y ? v : k;
  V* dst = blockIdx.y ? vc : kc;
  const long long sb = blockIdx.y ? v_sb : k_sb, sh = blockIdx.y ? v_sh : k_sh, ss = blockIdx.y ? v_ss : k_ss;
  for (long long i0 = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i0 < total; i0 += 4 * step) {
    V piece[4];
    long long at[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long i = i0 + u * step;       // (b, s, h, piece): the order of a projection's rows
      if (i >= total) continue;
      const int c = static_cast<int>(i % per);
      long long r = i / per;
      const int h = static_cast<int>(r % H);
      r /= H;
      const int s = static_cast<int>(r % S), b = static_cast<int>(r / S);
      piece[u] = src[b * sb + h * sh + s * ss + c];
      at[u] = ((static_cast<long long>(b) * H + h) * T + start + s) * per + c;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i0 + u * step < total) dst[at[u]] = piece[u];
  }
}

// Attention of one query per (row, head) over the cache. The splits of a row's keys are the CTAs of a cluster: they merge their
// (max, sum, output) through distributed shared memory, so there is no workspace and no second kernel.
// LPK lanes read a key (eight dims each) and a warp 32 / LPK keys at once, so a narrow head leaves no lane idle. Every lane fetches its
// own pieces of K and V with cp.async, DA_STAGES - 1 batches of DA_KEYS keys ahead: shared memory is a private queue, without barriers,
// and keeps up to 128 KB per SM on their way. With `k` given, the new token's key and value are rotated (the first rotary_dim
// dims), written to the cache at write_index[0] by the first split, and taken from registers by whichever split reaches that position.
// A write_index outside the cache writes nothing, makes the result NaN and sets the error word.
struct DecodeAttn {
  const void* q; const void* k; const void* v;          // [B, H, D] by strides (b, h); k, v may be null
  void* kc; void* vc; void* o;                          // caches [B, H, T, D], result [B, H, D]
  const int* lengths; const int* positions;             // keys per row, the new token's among them; its rotary position
  const long long* write_index;
  int* err;
  long long q_sb, q_sh, k_sb, k_sh, v_sb, v_sh;
  float scale, log2_base;
  int H, T, D, splits, window, rotary_dim;
};
constexpr int DA_WARPS = 4, DA_KEYS = 4, DA_STAGES = 3, DA_STAGE = 2 * DA_KEYS * 512 * DA_WARPS, DA_SMEM = DA_STAGES * DA_STAGE;
constexpr float DA_LOG2E = 1.4426950408889634f;

// 16 bytes into shared memory, or zeros where `live` is false (the address must be valid either way)
__device__ __forceinline__ void cp_piece(uint32_t dst, const void* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ uint4 ld_piece(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
  return v;
}
template <typename T> __device__ __forceinline__ void dec_unpack(const uint4& v, float (&f)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 t = DCvt<T>::to2(w[j]);
    f[2 * j] = t.x; f[2 * j + 1] = t.y;
  }
}
// eight dims from d0 on of a new q or k: rotated and rounded to T, as rotary_append_kernel stores them
template <typename T> __device__ __forceinline__ uint4 dec_rotate(const uint4& raw, int d0, int rotary_dim, float pos, float log2_base) {
  if (d0 >= rotary_dim) return raw;
  float f[8];
  dec_unpack<T>(raw, f);
  uint4 out;
  T* e = reinterpret_cast<T*>(&out);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int d = d0 + 2 * j;
    if (d < rotary_dim) {
      const float inv_freq = exp2f(-log2_base * static_cast<float>(d) / rotary_dim);
      float sn, cs;
      sincosf(pos * inv_freq, &sn, &cs);
      e[2 * j] = DCvt<T>::from(f[2 * j] * cs - f[2 * j + 1] * sn);
      e[2 * j + 1] = DCvt<T>::from(f[2 * j + 1] * cs + f[2 * j] * sn);
    } else {
      e[2 * j] = DCvt<T>::from(f[2 * j]);
      e[2 * j + 1] = DCvt<T>::from(f[2 * j + 1]);
    }
  }
  return out;
}

template <typename T, int LPK>
__global__ void __launch_bounds__(DA_WARPS * 32, 4) decode_attn_kernel(const DecodeAttn p) {
  constexpr int KPW = 32 / LPK, KB = DA_KEYS, DMAX = LPK * 8, BATCH = KB * KPW;
  extern __shared__ __align__(16) unsigned char da_smem[];
  __shared__ float red[DA_WARPS][DMAX];
  __shared__ float stat[DA_WARPS][2];
  __shared__ float fin[DMAX + 2];               // this split's output, maximum and sum
  const int sp = blockIdx.x, h = blockIdx.y, b = blockIdx.z, D = p.D;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, g = l / LPK, d0 = (l % LPK) * 8;
  const bool act = d0 < D;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  int len = p.lengths[b];
  if (len < 0 || len > p.T) {                   // a length that does not fit the cache: never read past it
    OSLO_REPORT_BOUNDS(p.err);
    len = len < 0 ? 0 : p.T;
  }
  const int lo = p.window > 0 ? max(0, len - p.window) : 0;
  const int span = len - lo, per = (span + p.splits - 1) / p.splits;
  const int t0 = lo + sp * per, t1 = min(len, t0 + per);
  const long long head = (static_cast<long long>(b) * p.H + h) * p.T * D;
  const T* kb = reinterpret_cast<const T*>(p.kc) + head + d0;
  const T* vb = reinterpret_cast<const T*>(p.vc) + head + d0;
  int wi = -1;
  if (p.k != nullptr) {
    const long long at = p.write_index[0];
    if (at >= 0 && at < p.T) wi = static_cast<int>(at);   // never write outside the cache
  }
  const uint32_t ring = smem_u32(da_smem) + (w * (2 * KB * 32) + l) * 16;
  int ft = t0 + w * BATCH, fslot = 0;
  auto fetch = [&]() {
    if (ft < t1) {
      const uint32_t at = ring + fslot * DA_STAGE;
#pragma unroll
      for (int j = 0; j < KB; ++j) {
        const int t = ft + j * KPW + g;
        const bool in = act && t < t1 && t != wi;
        const long long off = in ? static_cast<long long>(t) * D : -static_cast<long long>(d0);
        cp_piece(at + j * 512, kb + off, in);
        cp_piece(at + (KB + j) * 512, vb + off, in);
      }
    }
    ft += DA_WARPS * BATCH;
    if (++fslot == DA_STAGES) fslot = 0;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < DA_STAGES - 1; ++i) fetch();

  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 qraw = act ? *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.q) + b * p.q_sb + h * p.q_sh + d0) : zero;
  uint4 knew = zero, vnew = zero;
  if (p.k != nullptr) {
    if (act) {
      knew = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.k) + b * p.k_sb + h * p.k_sh + d0);
      vnew = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.v) + b * p.v_sb + h * p.v_sh + d0);
    }
    if (p.rotary_dim > 0) {
      const float pos = static_cast<float>(p.positions[b]);
      qraw = dec_rotate<T>(qraw, d0, p.rotary_dim, pos, p.log2_base);
      knew = dec_rotate<T>(knew, d0, p.rotary_dim, pos, p.log2_base);
    }
    if (wi >= 0 && sp == 0 && w == 0 && g == 0 && act) {
      *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.kc) + head + static_cast<long long>(wi) * D + d0) = knew;
      *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.vc) + head + static_cast<long long>(wi) * D + d0) = vnew;
    }
  }
  float q[8];
  dec_unpack<T>(qraw, q);
#pragma unroll
  for (int i = 0; i < 8; ++i) q[i] *= p.scale * DA_LOG2E;
  float m = -CUDART_INF_F, s = 0.f, acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  int slot = 0;
  for (int tb = t0 + w * BATCH; tb < t1; tb += DA_WARPS * BATCH) {
    fetch();                                    // into the slot of the batch before this one
    asm volatile("cp.async.wait_group %0;" ::"n"(DA_STAGES - 1) : "memory");
    const uint32_t at = ring + slot * DA_STAGE;
    if (++slot == DA_STAGES) slot = 0;
    uint4 kr[KB], vr[KB];
#pragma unroll
    for (int j = 0; j < KB; ++j) {
      kr[j] = ld_piece(at + j * 512);
      vr[j] = ld_piece(at + (KB + j) * 512);
    }
    if (wi >= tb && wi < tb + BATCH) {          // the batch that the new token falls into
#pragma unroll
      for (int j = 0; j < KB; ++j)
        if (tb + j * KPW + g == wi) { kr[j] = knew; vr[j] = vnew; }
    }
    float dot[KB];
#pragma unroll
    for (int j = 0; j < KB; ++j) {
      float f[8], d = 0.f;
      dec_unpack<T>(kr[j], f);
#pragma unroll
      for (int i = 0; i < 8; ++i) d += f[i] * q[i];
      dot[j] = d;
    }
#pragma unroll
    for (int off = LPK / 2; off > 0; off >>= 1) {
#pragma unroll
      for (int j = 0; j < KB; ++j) dot[j] += __shfl_xor_sync(0xffffffffu, dot[j], off);
    }
    float mn = m;
#pragma unroll
    for (int j = 0; j < KB; ++j) {
      if (tb + j * KPW + g >= t1) dot[j] = -CUDART_INF_F;
      mn = fmaxf(mn, dot[j]);
    }
    const float base = mn == -CUDART_INF_F ? 0.f : mn;   // this lane group may have no key in the batch
    const float a = exp2f(m - base);
    float ps = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] *= a;
#pragma unroll
    for (int j = 0; j < KB; ++j) {
      const float pr = exp2f(dot[j] - base);
      ps += pr;
      float f[8];
      dec_unpack<T>(vr[j], f);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += pr * f[i];
    }
    s = s * a + ps;
    m = mn;
  }
  // the lane groups of a warp, the warps of the block, the splits of the cluster
#pragma unroll
  for (int off = LPK; off < 32; off <<= 1) {
    const float mo = __shfl_xor_sync(0xffffffffu, m, off), so = __shfl_xor_sync(0xffffffffu, s, off);
    const float mx = fmaxf(m, mo), base = mx == -CUDART_INF_F ? 0.f : mx;
    const float a = exp2f(m - base), c = exp2f(mo - base);
    s = s * a + so * c;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = acc[i] * a + __shfl_xor_sync(0xffffffffu, acc[i], off) * c;
    m = mx;
  }
  if (l == 0) { stat[w][0] = m; stat[w][1] = s; }
  if (g == 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) red[w][d0 + i] = acc[i];
  }
  __syncthreads();
  float gm = -CUDART_INF_F, gs = 0.f, wt[DA_WARPS];
#pragma unroll
  for (int i = 0; i < DA_WARPS; ++i) gm = fmaxf(gm, stat[i][0]);
  {
    const float base = gm == -CUDART_INF_F ? 0.f : gm;
#pragma unroll
    for (int i = 0; i < DA_WARPS; ++i) { wt[i] = exp2f(stat[i][0] - base); gs += stat[i][1] * wt[i]; }
  }
  T* o = reinterpret_cast<T*>(p.o) + (static_cast<long long>(b) * p.H + h) * D;
  // a token that has no place in the cache: no answer from the keys that are left, and a report in every build (a replayed step has no
  // host to refuse it). Down here: in front of the loop it cost 4 % of a step of 32 rows
  const bool lost = p.k != nullptr && wi < 0;
  if (lost) {
    gs = CUDART_NAN_F;
    if (threadIdx.x == 0 && p.err != nullptr) atomicCAS(p.err, 0, ERR_BOUNDS);
  }
  for (int d = threadIdx.x; d < DMAX; d += DA_WARPS * 32) {
    float v = 0.f;
#pragma unroll
    for (int i = 0; i < DA_WARPS; ++i) v += red[i][d] * wt[i];
    if (p.splits > 1) fin[d] = v;
    else if (d < D) o[d] = DCvt<T>::from(gs > 0.f ? v / gs : (gs == gs ? 0.f : gs));
  }
  if (p.splits == 1) return;
  if (threadIdx.x == 0) { fin[DMAX] = gm; fin[DMAX + 1] = gs; }
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  const int share = (D + p.splits - 1) / p.splits;
  for (int dd = sp * share + threadIdx.x; dd < min(D, (sp + 1) * share); dd += DA_WARPS * 32) {
    const uint32_t base = smem_u32(fin);
    float pm[8], pv[8], psum[8], top = -CUDART_INF_F;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (r < p.splits) {
        uint32_t peer;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(base), "r"(r));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(pv[r]) : "r"(peer + dd * 4) : "memory");
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(pm[r]) : "r"(peer + DMAX * 4) : "memory");
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(psum[r]) : "r"(peer + (DMAX + 1) * 4) : "memory");
      } else {
        pv[r] = 0.f; pm[r] = -CUDART_INF_F; psum[r] = 0.f;
      }
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) top = fmaxf(top, pm[r]);
    const float ref = top == -CUDART_INF_F ? 0.f : top;
    float tot = 0.f, out = 0.f;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const float c = exp2f(pm[r] - ref);
      tot += psum[r] * c;
      out += pv[r] * c;
    }
    o[dd] = DCvt<T>::from(tot > 0.f ? out / tot : (tot == tot ? 0.f : tot));
  }
  // no block leaves while another may still read its part
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <typename T, int LPK>
static int decode_attn_launch(const DecodeAttn& p, int B, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(decode_attn_kernel<T, LPK>, cudaFuncAttributeMaxDynamicSharedMemorySize, DA_SMEM);
  if (e != cudaSuccess) return static_cast<int>(e);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.splits, p.H, B);
  cfg.blockDim = dim3(DA_WARPS * 32);
  cfg.dynamicSmemBytes = DA_SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.splits; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, decode_attn_kernel<T, LPK>, p));
}

template <typename T>
static int decode_attn_dispatch(const DecodeAttn& p, int B, cudaStream_t st) {
  if (p.D <= 32) return decode_attn_launch<T, 4>(p, B, st);
  if (p.D <= 64) return decode_attn_launch<T, 8>(p, B, st);
  if (p.D <= 128) return decode_attn_launch<T, 16>(p, B, st);
  return decode_attn_launch<T, 32>(p, B, st);
}

}  // namespace oslo

extern "C" int oslo_rotary_append(const void* q, const void* k, const void* v, long long ldq, long long ldk,
                                  long long ldv, void* q_out, void* kc, void* vc, const int* lengths,
                                  const long long* write_index, int B, int H, int D, int Tmax, int rotary_dim, float base,
                                  int dtype, int* err_word, cudaStream_t stream) {
  using namespace oslo;
  if (B <= 0 || H <= 0) return 0;
  if (D % 2 || rotary_dim % 2 || rotary_dim > D) return -1;
  dim3 grid(H, B);
  const int threads = D / 2 >= 128 ? 128 : (D / 2 >= 64 ? 64 : 32);
  if (dtype == OSLO_DT_BF16)
    rotary_append_kernel<__nv_bfloat16><<<grid, threads, 0, stream>>>(
        (const __nv_bfloat16*)q, (const __nv_bfloat16*)k, (const __nv_bfloat16*)v, ldq, ldk, ldv, (__nv_bfloat16*)q_out,
        (__nv_bfloat16*)kc, (__nv_bfloat16*)vc, lengths, write_index, H, D, Tmax, rotary_dim, log2f(base), err_word);
  else if (dtype == OSLO_DT_FP16)
    rotary_append_kernel<__half><<<grid, threads, 0, stream>>>((const __half*)q, (const __half*)k, (const __half*)v, ldq,
                                                               ldk, ldv, (__half*)q_out, (__half*)kc, (__half*)vc, lengths,
                                                               write_index, H, D, Tmax, rotary_dim, log2f(base), err_word);
  else
    return -2;
  return static_cast<int>(cudaGetLastError());
}

extern "C" int oslo_prompt_append(const void* k, const void* v, void* kc, void* vc, long long k_sb, long long k_sh, long long k_ss,
                                  long long v_sb, long long v_sh, long long v_ss, int B, int H, int S, int D, int T, int start,
                                  cudaStream_t st) {
  using namespace oslo;
  if (B <= 0 || H <= 0 || S <= 0 || D <= 0) return 0;
  if (D % 8 || start < 0 || start + S > T) return -1;
  const long long strides[6] = {k_sb, k_sh, k_ss, v_sb, v_sh, v_ss};
  for (long long s : strides)
    if (s % 8) return -1;
  const void* ptrs[4] = {k, v, kc, vc};
  for (const void* p : ptrs)
    if (reinterpret_cast<uintptr_t>(p) & 15) return -4;
  const int per = D / 8;
  const long long total = static_cast<long long>(B) * H * S * per;
  const long long blocks = (total + 1023) / 1024;
  prompt_append_kernel<uint4><<<dim3(static_cast<unsigned>(blocks < 148 * 32 ? blocks : 148 * 32), 2), 256, 0, st>>>(
      (const uint4*)k, (const uint4*)v, (uint4*)kc, (uint4*)vc, k_sb / 8, k_sh / 8, k_ss / 8, v_sb / 8, v_sh / 8, v_ss / 8, H, S, per, T,
      start, total);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int oslo_decode_attn(const void* q, const void* k, const void* v, void* kc, void* vc, void* o, long long q_sb,
                                long long q_sh, long long k_sb, long long k_sh, long long v_sb, long long v_sh, const int* lengths,
                                const int* positions, const long long* write_index, int B, int H, int T, int D, int rotary_dim,
                                float base, float scale, int window, int dtype, int num_sms, int* err_word, cudaStream_t st) {
  using namespace oslo;
  if (B <= 0 || H <= 0) return 0;
  if (D % 8 || D > 256 || D <= 0 || rotary_dim % 2 || rotary_dim > D || B > 65535 || H > 65535) return -3;
  const long long strides[6] = {q_sb, q_sh, k_sb, k_sh, v_sb, v_sh};
  for (int i = 0; i < (k ? 6 : 2); ++i)
    if (strides[i] % 8) return -1;
  const void* ptrs[5] = {q, k, v, kc, vc};
  for (const void* p : ptrs)
    if (reinterpret_cast<uintptr_t>(p) & 15) return -4;
  DecodeAttn p = {};
  p.q = q; p.k = k; p.v = v; p.kc = kc; p.vc = vc; p.o = o; p.lengths = lengths; p.positions = positions;
  p.write_index = write_index; p.err = err_word;
  p.q_sb = q_sb; p.q_sh = q_sh; p.k_sb = k_sb; p.k_sh = k_sh; p.v_sb = v_sb; p.v_sh = v_sh;
  p.scale = scale; p.log2_base = log2f(base); p.H = H; p.T = T; p.D = D; p.window = window; p.rotary_dim = k ? rotary_dim : 0;
  // Up to eight blocks per SM, two waves of the four that fit (8 rows x 16 heads x 2048 keys of 128: 29.5 us, 30.5 with one wave, and
  // 37 in blocks of eight warps with up to ten per SM; 32 x 16 x 1101 keys of 256: 105, 113, 111), clusters of at most eight, and no
  // split of fewer than 64 keys. The kernel before (4 to 16 of 32 lanes idle for narrow heads, one load deep, rotary, append and the
  // merge of the splits in kernels of their own) took 64.6 and 103.9 us for these.
  const int reach = window > 0 && window < T ? window : T;
  int splits = static_cast<int>(8ll * num_sms / (static_cast<long long>(B) * H));
  if (splits > reach / 64) splits = reach / 64;
  p.splits = splits < 1 ? 1 : (splits > 8 ? 8 : splits);
  if (dtype == OSLO_DT_BF16) return decode_attn_dispatch<__nv_bfloat16>(p, B, st);
  if (dtype == OSLO_DT_FP16) return decode_attn_dispatch<__half>(p, B, st);
  return -2;
}
