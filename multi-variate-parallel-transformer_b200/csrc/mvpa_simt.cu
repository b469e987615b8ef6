// fp32 CUDA-core kernels of Flash-MVPA: forward and the full backward.
//
// These serve element type fp32 (where tensor-core input rounding would break the
// 1e-4 relative tolerance) and every shape the tcgen05 kernels do not take.  They
// are tiled through shared memory and deterministic: no floating-point atomics
// anywhere, cross-tile sums go through per-tile partials.
//
// What bounds them: short sequences have few row tiles, so the longest CTA sets the time.  Hence sixteen rows per
// CTA, the column tiles of a row tile shared by four groups of warps, loads in flight under the products (fp32; the
// 16-bit types convert on the way and load in place), and no CTA-wide barrier in the loop.  fp32, against 32-row CTAs
// with synchronous loads and five barriers per tile (device time): forward B 1 H 4 T 32 C 16 D 64 18.1 against 71.0 us;
// B 1 H 4 Hkv 2 T 24 C 22 D 64 forward 21.4 / 76.5, query side with the relative scores and delta 41 / 109, key side
// 50 / 208, the rest 8 / 23 us.
//
// Math follows the reference forward (`attentions/attn.py:232-333`: base-2 online
// softmax, window zero-fill, time-block causal mask, L = m + log2 l) and backward
// (`attentions/attn.py:561-751` plus autograd through `_rel_bias`, `:1305-1314`).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>

#include <cooperative_groups.h>

#include "mvpa_common.cuh"
#include "tc_ptx.cuh"

namespace mvpa {
namespace {

constexpr int kThreads = 256;
constexpr int kMinRows = 16;    // fewest rows a CTA of the query-side backward takes
constexpr int kDrelSplit = 32;  // split-K factor of the relative-key gradient reduction

__device__ __forceinline__ bool in_window(int ti, int tk, int T, int window) {
  const int dt = ti - tk;
  return window <= 0 || (dt <= window && dt >= -window) || ti == T - 1;
}

// ---- building blocks of the tiled kernels --------------------------------------------------------
//
// A CTA owns BM = 8 * WPG rows (queries in the forward and the query-side backward, keys in the key-side
// one) and NG groups of WPG warps share its column tiles: group g takes tiles g, g + NG, ... with its own
// tile buffers, named barrier and partial results, which are merged once at the end.  A warp owns eight
// rows; its two half-warps hold four each and their 16 lanes spread over the columns of a tile, so a
// row's maximum is a four-step shuffle, a row's probabilities never leave the warp, and each product reads
// (4 + KN / 16) 16-byte words per 16 * KN / 4 multiply-adds.

// Group barrier: the WPG warps of group g.
template <int WPG>
__device__ __forceinline__ void group_sync(int g) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "n"(32 * WPG) : "memory");
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int n = valid ? 16 : 0;  // 0: the destination is zero-filled and nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <typename Tin>
__device__ __forceinline__ float4 load4(const Tin* p) {
  if constexpr (sizeof(Tin) == 4) {
    return *reinterpret_cast<const float4*>(p);
  } else {
    const uint2 w = *reinterpret_cast<const uint2*>(p);
    const Tin* e = reinterpret_cast<const Tin*>(&w);
    return make_float4(to_f32<Tin>(e[0]), to_f32<Tin>(e[1]), to_f32<Tin>(e[2]), to_f32<Tin>(e[3]));
  }
}

template <typename Tin>
__device__ __forceinline__ void store4(Tin* p, float4 v) {
  if constexpr (sizeof(Tin) == 4) {
    *reinterpret_cast<float4*>(p) = v;
  } else {
    uint2 w;
    Tin* e = reinterpret_cast<Tin*>(&w);
    e[0] = from_f32<Tin>(v.x); e[1] = from_f32<Tin>(v.y); e[2] = from_f32<Tin>(v.z); e[3] = from_f32<Tin>(v.w);
    *reinterpret_cast<uint2*>(p) = w;
  }
}

// ROWS rows of D elements from global (row stride `sn`, rows at or past n_rows read as zero) to shared memory
// (fp32, ld = D + 4), by THREADS threads of which this one is number `t`: asynchronous copies for fp32 (the
// caller commits and waits), converting loads otherwise.  Thread t writes the elements
// [(i * THREADS + t) * 4, +4) of the row-major tile, the same ones on every call.
template <typename Tin, int D, int ROWS, int THREADS>
__device__ __forceinline__ void load_rows(float* dst, const Tin* src, int64_t sn, int row0, int n_rows, int t) {
  constexpr int LD = D + 4;
#pragma unroll
  for (int i = 0; i < (ROWS * D / 4 + THREADS - 1) / THREADS; ++i) {
    const int idx = i * THREADS + t;
    if ((ROWS * D / 4) % THREADS != 0 && idx >= ROWS * D / 4) break;
    const int r = idx / (D / 4), d = (idx % (D / 4)) * 4;
    const bool in = row0 + r < n_rows;
    const Tin* s = src + (int64_t)(in ? row0 + r : 0) * sn + d;
    if constexpr (sizeof(Tin) == 4)
      cp_async16(dst + r * LD + d, s, in);
    else
      *reinterpret_cast<float4*>(dst + r * LD + d) = in ? load4<Tin>(s) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

__device__ __forceinline__ uint64_t ffma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// acc[a][j] = sum_d A[a][d] * B[tx + 16 j][d]: A points at this half-warp's four rows, both ld = D + 4.
// Packed multiply-adds over pairs of d: half the instructions of scalar ones, which leaves issue slots for the
// shared-memory loads.  The two halves of d are summed by themselves, because four chains of D / 4 terms round less than
// a scalar sum in groups of four does, and two chains of D / 2 more: output and dq at 4 x 4 tokens, D 64, against 64 bits,
// 1.14e-7 and 2.24e-7 with four chains, 1.21e-7 and 2.28e-7 in groups, 1.28e-7 and 2.49e-7 with two chains (which are 3 %
// faster in the forward of 32 x 16 tokens: 17.5 against 18.1 us).
template <int D, int KJ>
__device__ __forceinline__ void product_nt(const float* A, const float* B, int tx, float (&acc)[4][KJ]) {
  constexpr int LD = D + 4;
  const float* b0 = B + tx * LD;
  auto half = [&](int d0) {
    uint64_t s[4][KJ];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int j = 0; j < KJ; ++j) s[a][j] = 0ull;
#pragma unroll 4
    for (int dd = 0; dd < D / 2; dd += 4) {
      const int d = d0 + dd;
      ulonglong2 x[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) x[a] = *reinterpret_cast<const ulonglong2*>(A + a * LD + d);
#pragma unroll
      for (int j = 0; j < KJ; ++j) {
        const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(b0 + 16 * j * LD + d);
#pragma unroll
        for (int a = 0; a < 4; ++a) s[a][j] = ffma2(x[a].y, y.y, ffma2(x[a].x, y.x, s[a][j]));
      }
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int j = 0; j < KJ; ++j) {
        const float v = __uint_as_float((uint32_t)s[a][j]) + __uint_as_float((uint32_t)(s[a][j] >> 32));
        acc[a][j] = d0 == 0 ? v : acc[a][j] + v;
      }
  };
  half(0);
  half(D / 2);
}

// Columns of a row that a lane holds: VW = D / 16 of them, in pieces of up to four adjacent ones.
template <int D>
struct LaneCols {
  static constexpr int VW = D / 16;                 // 1, 2, 4, 8
  static constexpr int PW = VW < 4 ? VW : 4;        // piece width
  static constexpr int NP = VW / PW;                // pieces
  __device__ static int col(int tx, int p) { return tx * PW + 16 * PW * p; }
  __device__ static void load(const float* row, int tx, float (&v)[VW]) {
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      if constexpr (PW == 4) {
        const float4 w = *reinterpret_cast<const float4*>(row + col(tx, p));
        v[4 * p] = w.x; v[4 * p + 1] = w.y; v[4 * p + 2] = w.z; v[4 * p + 3] = w.w;
      } else if constexpr (PW == 2) {
        const float2 w = *reinterpret_cast<const float2*>(row + col(tx, p));
        v[0] = w.x; v[1] = w.y;
      } else {
        v[0] = row[col(tx, p)];
      }
    }
  }
  __device__ static void store(float* row, int tx, const float (&v)[VW]) {
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      if constexpr (PW == 4) *reinterpret_cast<float4*>(row + col(tx, p)) = make_float4(v[4 * p], v[4 * p + 1], v[4 * p + 2], v[4 * p + 3]);
      else if constexpr (PW == 2) *reinterpret_cast<float2*>(row + col(tx, p)) = make_float2(v[0], v[1]);
      else row[col(tx, p)] = v[0];
    }
  }
};

// out[a][lane's columns] += sum_c P[a][c] * B[c][columns]: P points at this half-warp's four rows (ld = KN + 4).
template <int D, int KN>
__device__ __forceinline__ void product_nn(const float* P, const float* B, int tx, float (&out)[4][D / 16]) {
  constexpr int LD = D + 4, VW = D / 16, LP = KN + 4;
#pragma unroll 2
  for (int c = 0; c < KN; c += 4) {
    float4 x[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) x[a] = *reinterpret_cast<const float4*>(P + a * LP + c);
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
      float y[VW];
      LaneCols<D>::load(B + (c + cc) * LD, tx, y);
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const float xv = cc == 0 ? x[a].x : cc == 1 ? x[a].y : cc == 2 ? x[a].z : x[a].w;
#pragma unroll
        for (int e = 0; e < VW; ++e) out[a][e] = fmaf(xv, y[e], out[a][e]);
      }
    }
  }
}

__device__ __forceinline__ float half_warp_max(float x) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}
__device__ __forceinline__ float half_warp_sum(float x) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Relative scores of the CTA's rows, all groups together: TB[r][s] = c2 (q_r + vt) . r_time[s] and
// CB[r][e] = c2 (q_r + z) . r_chan[e]  (`attentions/attn.py:1305-1314`, scaled like `:292,307`), for the
// `valid` rows that exist, TB with strides tb_r / tb_s.  QT and QC hold the rows with the two biases added; the
// relative keys pass through the groups' tile buffers `Kg`.
template <typename Tin, int D, int WPG, int NG, int KN>
__device__ __forceinline__ void rel_products(const Args& p, int hk, const float* QT, const float* QC, float* Kg,
                                             int valid, float* TB, int64_t tb_r, int64_t tb_s, float* CB, int g, int tg) {
  constexpr int LD = D + 4, KJ = KN / 16;
  const int lane = threadIdx.x & 31, tx = lane & 15, r0 = (tg >> 5) * 8 + (lane >> 4) * 4;
  const int nt = (p.T + KN - 1) / KN, nc = (p.C + KN - 1) / KN;
  for (int job = g; job < nt + nc; job += NG) {
    const bool is_t = job < nt;
    const int s0 = (is_t ? job : job - nt) * KN, n = is_t ? p.T : p.C;
    const Tin* src = is_t ? (const Tin*)p.rt + (int64_t)hk * p.T * D : (const Tin*)p.rc + (int64_t)hk * p.C * D;
    load_rows<Tin, D, KN, 32 * WPG>(Kg, src, D, s0, n, tg);
    cp_async_commit();
    cp_async_wait<0>();
    group_sync<WPG>(g);
    float acc[4][KJ];
    product_nt<D, KJ>((is_t ? QT : QC) + r0 * LD, Kg, tx, acc);
#pragma unroll
    for (int j = 0; j < KJ; ++j) {
      const int s = s0 + tx + 16 * j;
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        if (s < n && r0 + a < valid) {
          if (is_t) TB[(r0 + a) * tb_r + s * tb_s] = acc[a][j] * p.c2;
          else CB[(int64_t)(r0 + a) * n + s] = acc[a][j] * p.c2;
        }
      }
    }
    group_sync<WPG>(g);  // the buffer is free again
  }
}

// CTAs that a multiprocessor holds as far as shared memory goes, with room for `slots` floats of time and channel slots:
// two where they fit, which the compiler has to be told (at most 128 registers a thread), or it takes 160 and one CTA stays
// out: forward B 2 H 8 T 48 C 32 D 32 165 against 136 us, query side 352 against 258.
constexpr int resident_ctas(size_t fixed_floats, size_t slots) {
  return 2 * (fixed_floats + slots) * sizeof(float) + 2 * 1024 <= 233472 ? 2 : 1;
}

// ------------------------------- forward -------------------------------------

template <int D, int WPG, int NG, int KN>
constexpr size_t fwd_fixed_floats() {
  return (size_t)8 * WPG * (D + 4) + (size_t)NG * 2 * KN * (D + 4) + (size_t)NG * WPG * 8 * (KN + 4);
}

template <typename Tin, int D, int WPG, int NG, int KN>
__global__ void __launch_bounds__(32 * WPG * NG, resident_ctas(fwd_fixed_floats<D, WPG, NG, KN>(), 8 * WPG * 64))
simt_fwd_kernel(Args p) {
  ptx::griddep_wait();
  constexpr int LD = D + 4, KJ = KN / 16, BM = 8 * WPG, LP = KN + 4, VW = D / 16;
  constexpr int GT = 32 * WPG, CT = GT * NG;  // threads of a group, of the CTA
  static_assert(NG * KN >= 2 * BM, "the V buffers hold two copies of the rows during the prologue");
  extern __shared__ __align__(16) float smem[];
  float* Qs = smem;
  float* Kall = Qs + BM * LD;
  float* Vall = Kall + NG * KN * LD;
  float* Pall = Vall + NG * KN * LD;
  float* TBs = Pall + NG * WPG * 8 * LP;
  float* CBs = TBs + BM * p.T;
  float* QT = Vall;  // prologue only
  float* QC = QT + BM * LD;

  const int tid = threadIdx.x, lane = tid & 31, tx = lane & 15;
  const int g = tid / GT, tg = tid % GT;
  const int r0 = (tg >> 5) * 8 + (lane >> 4) * 4;  // first of this half-warp's four rows
  float* Ks = Kall + g * KN * LD;
  float* Vs = Vall + g * KN * LD;
  float* Ps = Pall + (tid >> 5) * 8 * LP + (lane >> 4) * 4 * LP;

  const int qt = gridDim.x - 1 - blockIdx.x;  // heaviest (latest) query tiles first
  const int bh = blockIdx.y, b = bh / p.H, h = bh % p.H, hk = h / p.g;
  const int m0 = qt * BM;                // first row of the tile inside this call's q / o / lse
  const int N = p.N, T = p.T, C = p.C;
  const int Nq = p.q_tn * C;             // rows of this call (a query time range, or all of N)
  const int row0 = p.q_t0 * C;           // token index of row 0
  const Tin* q = (const Tin*)p.q + b * p.q_sb + h * p.q_sh;
  const Tin* k = (const Tin*)p.k + b * p.k_sb + hk * p.k_sh;
  const Tin* v = (const Tin*)p.v + b * p.v_sb + hk * p.v_sh;
  const int valid = min(BM, Nq - m0);

  {  // rows with the three biases: QT, QC for the relative scores, Qs = (q + u) c2 (`attentions/attn.py:180-183`)
    const Tin *u = (const Tin*)p.u + hk * D, *vt = (const Tin*)p.vt + hk * D, *z = (const Tin*)p.z + hk * D;
    for (int idx = tid; idx < BM * D / 4; idx += CT) {
      const int r = idx / (D / 4), d = (idx % (D / 4)) * 4;
      const float4 x = r < valid ? load4<Tin>(q + (int64_t)(m0 + r) * p.q_sn + d) : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 bu = load4<Tin>(u + d), bt = load4<Tin>(vt + d), bz = load4<Tin>(z + d);
      *reinterpret_cast<float4*>(Qs + r * LD + d) =
          make_float4((x.x + bu.x) * p.c2, (x.y + bu.y) * p.c2, (x.z + bu.z) * p.c2, (x.w + bu.w) * p.c2);
      *reinterpret_cast<float4*>(QT + r * LD + d) = make_float4(x.x + bt.x, x.y + bt.y, x.z + bt.z, x.w + bt.w);
      *reinterpret_cast<float4*>(QC + r * LD + d) = make_float4(x.x + bz.x, x.y + bz.y, x.z + bz.z, x.w + bz.w);
    }
  }
  __syncthreads();
  rel_products<Tin, D, WPG, NG, KN>(p, hk, QT, QC, Ks, valid, TBs, T, 1, CBs, g, tg);

  // time step, channel and relative scores of the four rows (rows past the end take the last one's)
  int ti[4], ci[4];
  const float *tb[4], *cb[4];  // tb[a][t_k], cb[a][-|c_i - c_k|]
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int r = min(r0 + a, valid - 1), i = row0 + m0 + r;  // token index in the whole sequence
    ti[a] = i / C;
    ci[a] = i % C;
    tb[a] = TBs + r * T + (T - 1 - ti[a]);
    cb[a] = CBs + r * C + (C - 1);
  }
  const int t_first = (row0 + m0) / C, t_last = (row0 + m0 + valid - 1) / C;
  const int hi = min(N, (t_last + 1) * C);  // causal bound (`attentions/attn.py:102-104,125-127`)
  const int n_tiles = (hi + KN - 1) / KN;
  // every pair of the tile outside the content window: its product with K is not needed
  auto light = [&](int t) {
    return p.window > 0 && t_last != T - 1 && t_first - (min(N, (t + 1) * KN) - 1) / C > p.window;
  };
  auto fetch_k = [&](int t) {
    if (t < n_tiles && !light(t)) load_rows<Tin, D, KN, GT>(Ks, k, p.k_sn, t * KN, N, tg);
    cp_async_commit();
  };
  fetch_k(g);  // (the relative scores' last use of the buffer ended with a group barrier)
  __syncthreads();  // TBs / CBs are complete, QT / QC (the V buffers) are free

  int tk[KJ], ck[KJ];  // time step and channel of this lane's keys, carried from tile to tile
  const int step_t = NG * KN / C, step_c = NG * KN % C;
#pragma unroll
  for (int j = 0; j < KJ; ++j) {
    const int kk = g * KN + tx + 16 * j;
    tk[j] = kk / C;
    ck[j] = kk % C;
  }
  float m[4], l[4], o[4][VW];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    m[a] = -INFINITY;
    l[a] = 0.f;
#pragma unroll
    for (int e = 0; e < VW; ++e) o[a][e] = 0.f;
  }
  for (int t = g; t < n_tiles; t += NG) {
    const int n0 = t * KN;
    cp_async_wait<0>();
    group_sync<WPG>(g);  // K has arrived, every warp has left the previous tile's V
    load_rows<Tin, D, KN, GT>(Vs, v, p.v_sn, n0, N, tg);
    cp_async_commit();
    float s[4][KJ];
    if (light(t)) {
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int j = 0; j < KJ; ++j) s[a][j] = 0.f;
    } else {
      product_nt<D, KJ>(Qs + r0 * LD, Ks, tx, s);
    }
    float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int j = 0; j < KJ; ++j) {
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        float x = -INFINITY;
        if (tk[j] <= ti[a]) {  // (keys past the end lie past the last time step)
          x = in_window(ti[a], tk[j], T, p.window) ? s[a][j] : 0.f;
          x += tb[a][tk[j]] + cb[a][-abs(ci[a] - ck[j])];
        }
        s[a][j] = x;
        mx[a] = fmaxf(mx[a], x);
      }
      tk[j] += step_t;
      ck[j] += step_c;
      if (ck[j] >= C) { ck[j] -= C; ++tk[j]; }
    }
    // online softmax (`attentions/attn.py:309-315`); l stays a per-lane partial sum until the end
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const float m_new = fmaxf(m[a], half_warp_max(mx[a]));
      const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
      const float alpha = exp2f(m[a] - m_use);
      m[a] = m_new;
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < KJ; ++j) {
        const float pr = exp2f(s[a][j] - m_use);
        Ps[a * LP + tx + 16 * j] = pr;
        sum += pr;
      }
      l[a] = l[a] * alpha + sum;
#pragma unroll
      for (int e = 0; e < VW; ++e) o[a][e] *= alpha;
    }
    cp_async_wait<0>();
    group_sync<WPG>(g);  // V has arrived, every warp has left K
    fetch_k(t + NG);
    product_nn<D, KN>(Ps, Vs, tx, o);
    __syncwarp();
  }
  // merge the groups' partial results
  __syncthreads();
  float* Om = Kall;            // [NG][BM][LD]
  float* ml = Pall;            // [NG][BM][2]
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    LaneCols<D>::store(Om + (g * BM + r0 + a) * LD, tx, o[a]);
    const float ls = half_warp_sum(l[a]);
    if (tx == 0) {
      ml[(g * BM + r0 + a) * 2] = m[a];
      ml[(g * BM + r0 + a) * 2 + 1] = ls;
    }
  }
  __syncthreads();
  Tin* op = (Tin*)p.o + b * p.o_sb + h * p.o_sh;
  for (int idx = tid; idx < BM * D / 4; idx += CT) {
    const int r = idx / (D / 4), d = (idx % (D / 4)) * 4;
    if (r >= valid) continue;
    float mm = -INFINITY, ll = 0.f;
#pragma unroll
    for (int gg = 0; gg < NG; ++gg) mm = fmaxf(mm, ml[(gg * BM + r) * 2]);
    const float m_use = (mm == -INFINITY) ? 0.f : mm;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int gg = 0; gg < NG; ++gg) {
      const float w = exp2f(ml[(gg * BM + r) * 2] - m_use);
      const float4 y = *reinterpret_cast<const float4*>(Om + (gg * BM + r) * LD + d);
      ll += ml[(gg * BM + r) * 2 + 1] * w;
      x.x += y.x * w; x.y += y.y * w; x.z += y.z * w; x.w += y.w * w;
    }
    const float inv = 1.f / ll;
    store4<Tin>(op + (int64_t)(m0 + r) * p.o_sn + d, make_float4(x.x * inv, x.y * inv, x.z * inv, x.w * inv));
    if (d == 0 && p.lse != nullptr) p.lse[(int64_t)bh * Nq + m0 + r] = mm + log2f(ll);
  }
}

// ------------------------------- backward ------------------------------------

// Query side: one CTA per (BM query rows, b, h); the groups share the causal key tiles.  Recomputes
// P = exp2(S2 - L), forms dS, accumulates the content part of dQ and the per-row sums of dS by time slot and
// by key channel, then finishes dq = dS_w K + dTB r_time + dCB r_chan.  On the way it leaves behind what the
// other kernels need: the relative scores and delta (key side), the gradients of the relative scores
// (dr_time / dr_chan) and the column sums of the three parts of dq (du / dvt / dz).
template <int D, int WPG, int NG, int KN>
constexpr size_t dq_fixed_floats() {
  return (size_t)2 * 8 * WPG * (D + 4) + (size_t)NG * 2 * KN * (D + 4) + (size_t)NG * WPG * 8 * (KN + 4) + 16 * WPG;
}

// INS: the relative scores also sit in shared memory; otherwise they are read back from the workspace (long
// time or channel axes, where the two groups' slot sums fill the shared memory).
template <typename Tin, int D, int WPG, int NG, int KN, bool INS>
__global__ void __launch_bounds__(32 * WPG * NG, resident_ctas(dq_fixed_floats<D, WPG, NG, KN>(), 8 * WPG * (NG + INS) * 64))
simt_dq_kernel(BwdArgs bw) {
  ptx::griddep_wait();
  constexpr int LD = D + 4, KJ = KN / 16, BM = 8 * WPG, LP = KN + 4, VW = D / 16;
  constexpr int GT = 32 * WPG, CT = GT * NG;
  static_assert(NG * KN >= 2 * BM && KN >= BM, "aliased areas");
  const Args& p = bw.a;
  extern __shared__ __align__(16) float smem[];
  float* Qs = smem;                    // (q + u) c2
  float* Gs = Qs + BM * LD;            // dO rows
  float* Kall = Gs + BM * LD;
  float* Vall = Kall + NG * KN * LD;
  float* Pall = Vall + NG * KN * LD;   // dS, per warp
  float* lse_s = Pall + NG * WPG * 8 * LP;
  float* dl_s = lse_s + BM;
  const int N = p.N, T = p.T, C = p.C, TC = T + C;
  float* dTall = dl_s + BM;            // [NG][BM][T], by slot
  float* dCall = dTall + NG * BM * T;  // [NG][BM][C], by key channel
  float* TBs = dCall + NG * BM * C;    // [BM][T]   (INS)
  float* CBs = TBs + BM * T;           // [BM][C]   (INS)
  float* QT = Vall;                    // prologue only
  float* QC = QT + BM * LD;

  const int tid = threadIdx.x, lane = tid & 31, tx = lane & 15;
  const int g = tid / GT, tg = tid % GT;
  const int r0 = (tg >> 5) * 8 + (lane >> 4) * 4;
  float* Ks = Kall + g * KN * LD;
  float* Vs = Vall + g * KN * LD;
  float* Ds = Pall + (tid >> 5) * 8 * LP + (lane >> 4) * 4 * LP;
  float* dT = dTall + g * BM * T;
  float* dC = dCall + g * BM * C;

  const int qt = gridDim.x - 1 - blockIdx.x;
  const int bh = blockIdx.y, b = bh / p.H, h = bh % p.H, hk = h / p.g;
  const int m0 = qt * BM, valid = min(BM, N - m0);
  const Tin* q = (const Tin*)p.q + b * p.q_sb + h * p.q_sh;
  const Tin* k = (const Tin*)p.k + b * p.k_sb + hk * p.k_sh;
  const Tin* v = (const Tin*)p.v + b * p.v_sb + hk * p.v_sh;
  const Tin* gp = (const Tin*)bw.d_o + b * bw.do_sb + h * bw.do_sh;
  const Tin* op = (const Tin*)p.o + b * p.o_sb + h * p.o_sh;

  {
    const Tin *u = (const Tin*)p.u + hk * D, *vt = (const Tin*)p.vt + hk * D, *z = (const Tin*)p.z + hk * D;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int idx = tid; idx < BM * D / 4; idx += CT) {
      const int r = idx / (D / 4), d = (idx % (D / 4)) * 4;
      const float4 x = r < valid ? load4<Tin>(q + (int64_t)(m0 + r) * p.q_sn + d) : zero;
      const float4 bu = load4<Tin>(u + d), bt = load4<Tin>(vt + d), bz = load4<Tin>(z + d);
      *reinterpret_cast<float4*>(Qs + r * LD + d) =
          make_float4((x.x + bu.x) * p.c2, (x.y + bu.y) * p.c2, (x.z + bu.z) * p.c2, (x.w + bu.w) * p.c2);
      *reinterpret_cast<float4*>(QT + r * LD + d) = make_float4(x.x + bt.x, x.y + bt.y, x.z + bt.z, x.w + bt.w);
      *reinterpret_cast<float4*>(QC + r * LD + d) = make_float4(x.x + bz.x, x.y + bz.y, x.z + bz.z, x.w + bz.w);
      *reinterpret_cast<float4*>(Gs + r * LD + d) = r < valid ? load4<Tin>(gp + (int64_t)(m0 + r) * bw.do_sn + d) : zero;
    }
    // delta = sum_d dO O  (`attentions/attn.py:1213`): one warp per row
    for (int r = tid >> 5; r < BM; r += CT / 32) {
      float acc = 0.f;
      if (r < valid) {
        for (int d = lane * 4; d < D; d += 128) {
          const float4 x = load4<Tin>(gp + (int64_t)(m0 + r) * bw.do_sn + d), y = load4<Tin>(op + (int64_t)(m0 + r) * p.o_sn + d);
          acc += x.x * y.x + x.y * y.y + x.z * y.z + x.w * y.w;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) {
        dl_s[r] = acc;
        lse_s[r] = r < valid ? p.lse[(int64_t)bh * N + m0 + r] : INFINITY;  // P = 0 on rows that do not exist
        if (r < valid) bw.delta[(int64_t)bh * N + m0 + r] = acc;
      }
    }
    for (int idx = tid; idx < NG * BM * TC; idx += CT) dTall[idx] = 0.f;  // dTall and dCall are adjacent
  }
  __syncthreads();
  // the relative scores, time slots row-innermost and channel slots as they are: the key side reads them too
  float* tbg = bw.tbg + (int64_t)bh * N * T + m0;
  float* cbg = bw.cbg + ((int64_t)bh * N + m0) * C;
  if constexpr (INS) rel_products<Tin, D, WPG, NG, KN>(p, hk, QT, QC, Ks, valid, TBs, T, 1, CBs, g, tg);
  else rel_products<Tin, D, WPG, NG, KN>(p, hk, QT, QC, Ks, valid, tbg, 1, N, cbg, g, tg);

  int ti[4], ci[4];
  const float *tb[4], *cb[4];  // the scores of the four rows (rows past the end take the last one's)
  const int64_t tb_s = INS ? 1 : N;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int r = min(r0 + a, valid - 1), i = m0 + r;
    ti[a] = i / C;
    ci[a] = i % C;
    tb[a] = (INS ? TBs + r * T : tbg + r) + (T - 1 - ti[a]) * tb_s;
    cb[a] = (INS ? CBs : cbg) + (int64_t)r * C + (C - 1);
  }
  const int t_first = m0 / C, t_last = (m0 + valid - 1) / C;
  const int hi = min(N, (t_last + 1) * C);
  const int n_tiles = (hi + KN - 1) / KN;
  auto light = [&](int t) {
    return p.window > 0 && t_last != T - 1 && t_first - (min(N, (t + 1) * KN) - 1) / C > p.window;
  };
  auto fetch_k = [&](int t) {
    if (t < n_tiles && !light(t)) load_rows<Tin, D, KN, GT>(Ks, k, p.k_sn, t * KN, N, tg);
    cp_async_commit();
  };
  auto fetch_v = [&](int t) {
    if (t < n_tiles) load_rows<Tin, D, KN, GT>(Vs, v, p.v_sn, t * KN, N, tg);
    cp_async_commit();
  };
  __syncthreads();  // TBs / CBs are complete, QT / QC (the V buffers) are free
  fetch_v(g);
  fetch_k(g);
  if constexpr (INS) {
    for (int idx = tid; idx < BM * T; idx += CT) {
      const int r = idx % BM, s = idx / BM;
      if (r < valid) tbg[(int64_t)s * N + r] = TBs[r * T + s];
    }
    for (int idx = tid; idx < valid * C; idx += CT) cbg[idx] = CBs[idx];
  }

  int tk[KJ], ck[KJ];  // time step and channel of this lane's keys, carried from tile to tile
  const int step_t = NG * KN / C, step_c = NG * KN % C;
#pragma unroll
  for (int j = 0; j < KJ; ++j) {
    const int kk = g * KN + tx + 16 * j;
    tk[j] = kk / C;
    ck[j] = kk % C;
  }
  float acc[4][VW], lse[4], dl[4];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    lse[a] = lse_s[r0 + a];
    dl[a] = dl_s[r0 + a];
#pragma unroll
    for (int e = 0; e < VW; ++e) acc[a][e] = 0.f;
  }
  for (int t = g; t < n_tiles; t += NG) {
    const int n0 = t * KN;
    const bool lt = light(t);
    cp_async_wait<1>();
    group_sync<WPG>(g);  // V has arrived
    float s[4][KJ], dp[4][KJ];
    product_nt<D, KJ>(Gs + r0 * LD, Vs, tx, dp);
    cp_async_wait<0>();
    group_sync<WPG>(g);  // K has arrived, every warp has left V
    fetch_v(t + NG);
    if (lt) {
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int j = 0; j < KJ; ++j) s[a][j] = 0.f;
    } else {
      product_nt<D, KJ>(Qs + r0 * LD, Ks, tx, s);
    }
    bool w[4][KJ];
#pragma unroll
    for (int j = 0; j < KJ; ++j) {
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        float ds = 0.f;
        w[a][j] = in_window(ti[a], tk[j], T, p.window);
        if (tk[j] <= ti[a]) {  // (keys past the end lie past the last time step)
          const float s2 = (w[a][j] ? s[a][j] : 0.f) + tb[a][tk[j] * tb_s] + cb[a][-abs(ci[a] - ck[j])];
          ds = exp2f(s2 - lse[a]) * (dp[a][j] - dl[a]) * p.sm_scale;  // `attentions/attn.py:680`
        }
        s[a][j] = ds;
        Ds[a * LP + tx + 16 * j] = ds;
      }
      tk[j] += step_t;
      ck[j] += step_c;
      if (ck[j] >= C) { ck[j] -= C; ++tk[j]; }
    }
    __syncwarp();
    {  // sums of dS over the tile, by key time step (the reference's dS x csm_time product, `:681-694`) and by
       // key channel; this half-warp's lanes take the (row, time step) and (row, channel) pairs of its rows
      const int last = min(n0 + KN, N) - 1, tk0 = n0 / C, tk1 = last / C, nT = tk1 - tk0 + 1;
      for (int idx = tx; idx < 4 * nT; idx += 16) {
        const int a = idx & 3, tk = tk0 + (idx >> 2);
        const int t_i = min(m0 + r0 + a, N - 1) / C;
        if (tk <= t_i) {
          const int lo = max(n0, tk * C) - n0, up = min(last, tk * C + C - 1) - n0;
          float sum = 0.f;
          for (int c = lo; c <= up; ++c) sum += Ds[a * LP + c];
          dT[(r0 + a) * T + (T - 1 - (t_i - tk))] += sum;
        }
      }
      const int c_n = min(C, last - n0 + 1), c_b = n0 - tk0 * C;  // distinct channels of the tile, the first one
      for (int idx = tx; idx < 4 * c_n; idx += 16) {
        const int a = idx & 3, off = idx >> 2;
        float sum = 0.f;
        for (int c = off; c <= last - n0; c += C) sum += Ds[a * LP + c];
        int ch = c_b + off;
        if (ch >= C) ch -= C;
        dC[(r0 + a) * C + ch] += sum;
      }
    }
    __syncwarp();
    if (!lt) {  // dQ += dS_w K   (`attentions/attn.py:708-730`)
#pragma unroll
      for (int j = 0; j < KJ; ++j)
#pragma unroll
        for (int a = 0; a < 4; ++a)
          if (!w[a][j]) Ds[a * LP + tx + 16 * j] = 0.f;
      __syncwarp();
      product_nn<D, KN>(Ds, Ks, tx, acc);
    }
    group_sync<WPG>(g);  // every warp has left K
    fetch_k(t + NG);
  }
  __syncthreads();
  // merge: dq's content part of every group, the slot sums, channel sums folded by |c_i - c_k| (`:695-707`)
  float* Am = Kall;  // [NG][BM][LD]
#pragma unroll
  for (int a = 0; a < 4; ++a) LaneCols<D>::store(Am + (g * BM + r0 + a) * LD, tx, acc[a]);
  float* dtbg = bw.dtbg + ((int64_t)bh * N + m0) * T;
  for (int idx = tid; idx < BM * T; idx += CT) {
    float s = 0.f;
#pragma unroll
    for (int gg = 0; gg < NG; ++gg) s += dTall[gg * BM * T + idx];
    dTall[idx] = s;
    if (idx < valid * T) dtbg[idx] = s;
  }
  float* dcbg = bw.dcbg + ((int64_t)bh * N + m0) * C;
  for (int idx = tid; idx < BM * C; idx += CT) {
    const int r = idx / C, e = C - 1 - (idx - r * C), c_i = min(m0 + r, N - 1) % C;
    float s = 0.f;
#pragma unroll
    for (int gg = 0; gg < NG; ++gg) {
      const float* row = dCall + (gg * BM + r) * C;
      if (c_i - e >= 0) s += row[c_i - e];
      if (e > 0 && c_i + e < C) s += row[c_i + e];
    }
    if constexpr (INS) CBs[idx] = s;  // (the scores have been used)
    if (r < valid) dcbg[idx] = s;
  }
  __syncthreads();
  // dq = content + dTB r_time + dCB r_chan (autograd through `_rel_bias`); a thread holds four columns of a row
  float* parts = Vall;  // [2][BM][LD]: the temporal and the channel part; the content part replaces Am's first copy
  const Tin* rt = (const Tin*)p.rt + (int64_t)hk * T * D;
  const Tin* rc = (const Tin*)p.rc + (int64_t)hk * C * D;
  Tin* dq = (Tin*)bw.dq + b * bw.dq_sb + h * bw.dq_sh;
  for (int idx = tid; idx < BM * D / 4; idx += CT) {
    const int r = idx / (D / 4), d = (idx % (D / 4)) * 4;
    float4 x = *reinterpret_cast<const float4*>(Am + r * LD + d);
#pragma unroll
    for (int gg = 1; gg < NG; ++gg) {
      const float4 y = *reinterpret_cast<const float4*>(Am + (gg * BM + r) * LD + d);
      x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w;
    }
    float4 part[2];
#pragma unroll
    for (int which = 0; which < 2; ++which) {
      const int n = which == 0 ? T : C;
      const float* f = (which == 0 ? dTall : INS ? CBs : dcbg) + (int64_t)(which == 0 || INS ? r : min(r, valid - 1)) * n;
      const Tin* key = (which == 0 ? rt : rc) + d;
      float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
      for (int s = 0; s < (r < valid ? n : 0); ++s) {  // (rows past the end: zero)
        const float4 kv = load4<Tin>(key + (int64_t)s * D);
        const float fv = f[s];
        y.x = fmaf(fv, kv.x, y.x); y.y = fmaf(fv, kv.y, y.y); y.z = fmaf(fv, kv.z, y.z); y.w = fmaf(fv, kv.w, y.w);
      }
      part[which] = y;
      *reinterpret_cast<float4*>(parts + (which * BM + r) * LD + d) = y;
    }
    *reinterpret_cast<float4*>(Am + r * LD + d) = x;
    if (r < valid)
      store4<Tin>(dq + (int64_t)(m0 + r) * bw.dq_sn + d,
                  make_float4(x.x + part[0].x + part[1].x, x.y + part[0].y + part[1].y, x.z + part[0].z + part[1].z,
                              x.w + part[0].w + part[1].w));
  }
  __syncthreads();
  // column sums; rows past the end contributed zeros everywhere
  float* out = bw.partial + ((int64_t)bh * gridDim.x + qt) * 3 * D;
  for (int idx = tid; idx < 3 * D; idx += CT) {
    const int which = idx / D, d = idx % D;
    const float* src = (which == 0 ? Am : parts + (which - 1) * BM * LD) + d;
    float s = 0.f;
#pragma unroll
    for (int r = 0; r < BM; ++r) s += src[r * LD];
    out[idx] = s;
  }
}

// Key side: one CTA per (BM keys, b, kv head); the groups share the (query head of the group, causal query
// tile) items.  Products are formed transposed (key rows x query columns).
template <int D, int WPG, int NG, int KN>
constexpr size_t dkv_fixed_floats() {
  return (size_t)2 * 8 * WPG * (D + 4) + (size_t)NG * 2 * KN * (D + 4) + (size_t)NG * WPG * 16 * (KN + 4) + 2 * NG * KN;
}

// (two CTAs a multiprocessor at D 16: 159 against 185 us at B 2 H 8 T 48 C 32; from D 32 on the 128 registers that leaves
// a thread spill: 387 against 232 us)
template <typename Tin, int D, int WPG, int NG, int KN>
__global__ void __launch_bounds__(32 * WPG * NG, D == 16 ? 2 : 1) simt_dkv_kernel(BwdArgs bw) {
  ptx::griddep_wait();
  constexpr int LD = D + 4, KJ = KN / 16, BM = 8 * WPG, LP = KN + 4, VW = D / 16;
  constexpr int GT = 32 * WPG, CT = GT * NG;
  static_assert(KN >= BM, "aliased areas");
  const Args& p = bw.a;
  extern __shared__ __align__(16) float smem[];
  float* Ks = smem;
  float* Vs = Ks + BM * LD;
  float* Qall = Vs + BM * LD;
  float* Gall = Qall + NG * KN * LD;
  float* Pall = Gall + NG * KN * LD;      // P^T and dS_w^T of each warp's eight key rows
  float* Lall = Pall + NG * WPG * 16 * LP;  // log-sum-exp and delta of each group's query tile

  const int tid = threadIdx.x, lane = tid & 31, tx = lane & 15;
  const int g = tid / GT, tg = tid % GT;
  const int r0 = (tg >> 5) * 8 + (lane >> 4) * 4;
  float* Qs = Qall + g * KN * LD;
  float* Gs = Gall + g * KN * LD;
  float* Ps = Pall + (tid >> 5) * 16 * LP + (lane >> 4) * 4 * LP;
  float* Dw = Ps + 8 * LP;
  float* lse_s = Lall + g * 2 * KN;
  float* dl_s = lse_s + KN;

  const int bk = blockIdx.y, b = bk / p.Hkv, hk = bk % p.Hkv;
  const int n0 = blockIdx.x * BM;  // earliest keys (seen by the most queries) first
  const int N = p.N, T = p.T, C = p.C;
  const int valid = min(BM, N - n0);
  load_rows<Tin, D, BM, CT>(Ks, (const Tin*)p.k + b * p.k_sb + hk * p.k_sh, p.k_sn, n0, N, tid);
  load_rows<Tin, D, BM, CT>(Vs, (const Tin*)p.v + b * p.v_sb + hk * p.v_sh, p.v_sn, n0, N, tid);
  cp_async_commit();
  int tk[4], ck[4];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int kk = min(n0 + r0 + a, N - 1);
    tk[a] = kk / C;
    ck[a] = kk % C;
  }
  const int tk_last = (n0 + valid - 1) / C;
  const int tile0 = ((n0 / C) * C) / KN, per_head = (N + KN - 1) / KN - tile0;  // first query tile that sees these keys
  const int items = p.g * per_head;
  // The CTAs of a cluster (gridDim.z of them own the same keys) and their groups take the items in turn.
  const int part = blockIdx.z, parts = gridDim.z, first = part * NG + g, stride = parts * NG;
  // every pair outside the content window: neither S nor dS_w is needed, only P
  auto light = [&](int m0) {
    const int t_hi = (min(N, m0 + KN) - 1) / C;
    return p.window > 0 && t_hi != T - 1 && m0 / C - tk_last > p.window;
  };
  const float4 u4 = load4<Tin>((const Tin*)p.u + hk * D + (tg % (D / 4)) * 4);  // bias of the columns this thread loads
  static_assert(GT % (D / 4) == 0, "a thread loads the same columns of every row");
  auto fetch_q = [&](int item) {
    if (item < items) {
      const int h = hk * p.g + item / per_head, m0 = (tile0 + item % per_head) * KN;
      if (!light(m0)) load_rows<Tin, D, KN, GT>(Qs, (const Tin*)p.q + b * p.q_sb + h * p.q_sh, p.q_sn, m0, N, tg);
    }
    cp_async_commit();
  };
  auto fetch_g = [&](int item) {
    if (item < items) {
      const int h = hk * p.g + item / per_head, m0 = (tile0 + item % per_head) * KN;
      load_rows<Tin, D, KN, GT>(Gs, (const Tin*)bw.d_o + b * bw.do_sb + h * bw.do_sh, bw.do_sn, m0, N, tg);
    }
    cp_async_commit();
  };
  float kacc[4][VW], vacc[4][VW];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int e = 0; e < VW; ++e) kacc[a][e] = vacc[a][e] = 0.f;
  fetch_q(first);
  fetch_g(first);
  cp_async_wait<2>();
  __syncthreads();  // K and V are in place
  for (int item = first; item < items; item += stride) {
    const int h = hk * p.g + item / per_head, bh = b * p.H + h, m0 = (tile0 + item % per_head) * KN;
    const bool lt = light(m0);
    const float* tbg = bw.tbg + (int64_t)bh * N * T;
    const float* cbg = bw.cbg + (int64_t)bh * N * C;
    // this tile's relative scores, requested before the products that hide their latency
    float rel[4][KJ];
    int ti[KJ];
#pragma unroll
    for (int j = 0; j < KJ; ++j) {
      const int i = min(m0 + tx + 16 * j, N - 1), t_i = i / C, c_i = i % C;
      ti[j] = t_i;
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const int dt = max(t_i - tk[a], 0);
        rel[a][j] = tbg[(int64_t)(T - 1 - dt) * N + i] + cbg[(int64_t)i * C + (C - 1 - abs(c_i - ck[a]))];
      }
    }
    for (int c = tg; c < KN; c += GT) {
      const int i = min(m0 + c, N - 1);
      lse_s[c] = p.lse[(int64_t)bh * N + i];
      dl_s[c] = bw.delta[(int64_t)bh * N + i];
    }
    cp_async_wait<1>();  // Q: this thread's own pieces
    if (!lt) {           // Q <- (q + u) c2, rows past the end included (their P is 0)
#pragma unroll
      for (int i = 0; i < KN * D / 4 / GT; ++i) {
        const int idx = i * GT + tg;
        float4* x = reinterpret_cast<float4*>(Qs + (idx / (D / 4)) * LD + (idx % (D / 4)) * 4);
        const float4 y = *x;
        *x = make_float4((y.x + u4.x) * p.c2, (y.y + u4.y) * p.c2, (y.z + u4.z) * p.c2, (y.w + u4.w) * p.c2);
      }
    }
    cp_async_wait<0>();
    group_sync<WPG>(g);  // Q, dO, lse and delta are in place
    float s[4][KJ], dp[4][KJ];
    if (lt) {
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int j = 0; j < KJ; ++j) s[a][j] = dp[a][j] = 0.f;
    } else {
      product_nt<D, KJ>(Ks + r0 * LD, Qs, tx, s);   // S^T in base 2 (Q carries c2)
      product_nt<D, KJ>(Vs + r0 * LD, Gs, tx, dp);  // dP^T
    }
#pragma unroll
    for (int j = 0; j < KJ; ++j) {
      const int col = tx + 16 * j, i = m0 + col, t_i = ti[j];
      const float lse = lse_s[col], dl = dl_s[col];
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        float pr = 0.f, dsw = 0.f;
        if (i < N && tk[a] <= t_i) {
          const bool w = in_window(t_i, tk[a], T, p.window);
          pr = exp2f((w ? s[a][j] : 0.f) + rel[a][j] - lse);
          dsw = w ? pr * (dp[a][j] - dl) * p.sm_scale : 0.f;
        }
        Ps[a * LP + col] = pr;
        Dw[a * LP + col] = dsw;
      }
    }
    __syncwarp();
    if (!lt) product_nn<D, KN>(Dw, Qs, tx, kacc);  // dK += dS_w^T (q + u) c2  (`attentions/attn.py:718`)
    group_sync<WPG>(g);                            // every warp has left Q, lse and delta
    fetch_q(item + stride);
    product_nn<D, KN>(Ps, Gs, tx, vacc);           // dV += P^T dO        (`attentions/attn.py:671-675`)
    group_sync<WPG>(g);                            // every warp has left dO
    fetch_g(item + stride);
  }
  __syncthreads();
  float *Km = Qall, *Vm = Gall;  // [NG][BM][LD] each
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    LaneCols<D>::store(Km + (g * BM + r0 + a) * LD, tx, kacc[a]);
    LaneCols<D>::store(Vm + (g * BM + r0 + a) * LD, tx, vacc[a]);
  }
  __syncthreads();
  Tin* dk = (Tin*)bw.dk + b * bw.dk_sb + hk * bw.dk_sh;
  Tin* dv = (Tin*)bw.dv + b * bw.dv_sb + hk * bw.dv_sh;
  const float inv_c2 = 1.f / p.c2;
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  if (parts > 1) cluster.sync();  // every CTA's sums are in its shared memory
  for (int idx = part * CT + tid; idx < 2 * BM * D / 4; idx += parts * CT) {
    const bool is_k = idx < BM * D / 4;
    const int rem = is_k ? idx : idx - BM * D / 4;
    const int r = rem / (D / 4), d = (rem % (D / 4)) * 4;
    if (r >= valid) continue;
    float* own = (is_k ? Km : Vm) + r * LD + d;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int q = 0; q < parts; ++q) {
      const float* src = parts > 1 ? cluster.map_shared_rank(own, q) : own;
      float4 z = *reinterpret_cast<const float4*>(src);
#pragma unroll
      for (int gg = 1; gg < NG; ++gg) {
        const float4 y = *reinterpret_cast<const float4*>(src + gg * BM * LD);
        z.x += y.x; z.y += y.y; z.z += y.z; z.w += y.w;
      }
      if (q == 0) x = z;
      else { x.x += z.x; x.y += z.y; x.z += z.z; x.w += z.w; }
    }
    if (is_k)
      store4<Tin>(dk + (int64_t)(n0 + r) * bw.dk_sn + d, make_float4(x.x * inv_c2, x.y * inv_c2, x.z * inv_c2, x.w * inv_c2));
    else
      store4<Tin>(dv + (int64_t)(n0 + r) * bw.dv_sn + d, x);
  }
  if (parts > 1) cluster.sync();  // nobody leaves while its sums are still being read
}

// dr[hk][slot][d] = sum_{b, h in group, i} dX[b,h,i,slot] * (q[b,h,i,d] + bias[hk][d]), for the T time slots and
// the C channel slots in one launch.  One CTA per (32 slots, kv head, split); streams its share of the group's
// query rows in chunks of 64.
constexpr int kDrelRows = 64, kDrelSlots = 32;
template <typename Tin, int D>
__global__ void __launch_bounds__(kThreads) simt_drel_kernel(BwdArgs bw) {
  ptx::griddep_wait();
  constexpr int LD = D + 4, VW = D / 16, LX = kDrelSlots + 1;
  const Args& p = bw.a;
  extern __shared__ __align__(16) float smem[];
  float* Qs = smem;                  // 64 rows x LD
  float* Xs = Qs + kDrelRows * LD;   // 64 rows x 33
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int t_blocks = (p.T + kDrelSlots - 1) / kDrelSlots;
  const bool is_t = (int)blockIdx.x < t_blocks;
  const int S = is_t ? p.T : p.C, s0 = (is_t ? blockIdx.x : blockIdx.x - t_blocks) * kDrelSlots;
  const float* dx = is_t ? bw.dtbg : bw.dcbg;
  const int hk = blockIdx.y;
  const Tin* bias = (const Tin*)(is_t ? p.vt : p.z) + hk * D;
  // split-K over the (batch, head of the group, 64-row chunk) range: gridDim.z partial sums
  float* out = bw.drel_part + (((int64_t)blockIdx.z * p.Hkv + hk) * (p.T + p.C) + (is_t ? 0 : p.T)) * D;
  const int chunks_per_head = (p.N + kDrelRows - 1) / kDrelRows;
  const int n_chunks = p.B * p.g * chunks_per_head;
  const int per_z = (n_chunks + gridDim.z - 1) / gridDim.z;
  const int c_begin = blockIdx.z * per_z, c_end = min(n_chunks, c_begin + per_z);
  float acc[2][VW] = {};
  for (int ch = c_begin; ch < c_end; ++ch) {
    const int b = ch / (p.g * chunks_per_head), hh = (ch / chunks_per_head) % p.g;
    const int m0 = (ch % chunks_per_head) * kDrelRows;
    const int h = hk * p.g + hh, bh = b * p.H + h;
    const Tin* q = (const Tin*)p.q + b * p.q_sb + h * p.q_sh;
    __syncthreads();
#pragma unroll
    for (int idx = tid; idx < kDrelRows * D / 4; idx += kThreads) {
      const int r = idx / (D / 4), d = (idx % (D / 4)) * 4;
      const float4 bb = load4<Tin>(bias + d);
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (m0 + r < p.N) x = load4<Tin>(q + (int64_t)(m0 + r) * p.q_sn + d);
      *reinterpret_cast<float4*>(Qs + r * LD + d) = make_float4(x.x + bb.x, x.y + bb.y, x.z + bb.z, x.w + bb.w);
    }
#pragma unroll
    for (int idx = tid; idx < kDrelRows * kDrelSlots; idx += kThreads) {
      const int r = idx / kDrelSlots, s = idx % kDrelSlots;
      const int i = m0 + r;
      Xs[r * LX + s] = (i < p.N && s0 + s < S) ? dx[((int64_t)bh * p.N + i) * S + s0 + s] : 0.f;
    }
    __syncthreads();
    // rows past the end hold the bias alone in Qs but zero in Xs, so they add nothing
#pragma unroll 8
    for (int r = 0; r < kDrelRows; ++r) {
      const float x0 = Xs[r * LX + 2 * ty], x1 = Xs[r * LX + 2 * ty + 1];
      float y[VW];
      LaneCols<D>::load(Qs + r * LD, tx, y);
#pragma unroll
      for (int e = 0; e < VW; ++e) {
        acc[0][e] = fmaf(x0, y[e], acc[0][e]);
        acc[1][e] = fmaf(x1, y[e], acc[1][e]);
      }
    }
  }
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    const int s = s0 + 2 * ty + a;
    if (s < S) LaneCols<D>::store(out + (int64_t)s * D, tx, acc[a]);
  }
}

// The last sums, in a fixed order (deterministic): dr_time / dr_chan from the split-K partials of
// simt_drel_kernel (the first n_red blocks), du / dvt / dz from the per-tile partials of simt_dq_kernel (three
// blocks per kv head).
__global__ void __launch_bounds__(kThreads) simt_final_kernel(BwdArgs bw, int n_z, int n_qt, int n_red) {
  ptx::griddep_wait();
  const Args& p = bw.a;
  const int S = p.T + p.C, D = p.D;
  if ((int)blockIdx.x < n_red) {
    const int64_t total = (int64_t)p.Hkv * S * D;
    for (int64_t idx = (int64_t)blockIdx.x * kThreads + threadIdx.x; idx < total; idx += (int64_t)n_red * kThreads) {
      float sum = 0.f;
#pragma unroll 8
      for (int zz = 0; zz < n_z; ++zz) sum += bw.drel_part[(int64_t)zz * total + idx];
      const int d = idx % D, sl = (idx / D) % S, hk = idx / ((int64_t)D * S);
      if (sl < p.T) bw.drt[((int64_t)hk * p.T + sl) * D + d] = sum;
      else bw.drc[((int64_t)hk * p.C + (sl - p.T)) * D + d] = sum;
    }
    return;
  }
  __shared__ float s_part[kThreads];
  const int hk = ((int)blockIdx.x - n_red) / 3, which = ((int)blockIdx.x - n_red) % 3;
  const int d = threadIdx.x % D, part = threadIdx.x / D, parts = kThreads / D;  // D divides the block size
  const int per_b = p.g * n_qt, n = p.B * per_b;
  float s = 0.f;
#pragma unroll 8
  for (int it = part; it < n; it += parts) {
    const int b = it / per_b;
    const int64_t tile = ((int64_t)b * p.H + hk * p.g) * n_qt + (it - b * per_b);
    s += bw.partial[(tile * 3 + which) * D + d];
  }
  s_part[threadIdx.x] = s;
  __syncthreads();
  if (part == 0) {
    for (int q = 1; q < parts; ++q) s += s_part[q * D + d];
    float* out = which == 0 ? bw.du : which == 1 ? bw.dvt : bw.dz;
    out[hk * D + d] = s;
  }
}

template <typename K>
int set_smem(K kernel, size_t bytes) {
  if (bytes > 48 * 1024) {
    MVPA_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  }
  return MVPA_OK;
}

constexpr size_t kMaxSmemFloats = 232448 / sizeof(float);

// Rows per CTA and groups: sixteen rows and four groups while that leaves no more than kSmallWaves CTAs per
// multiprocessor (short sequences: the longest CTA sets the time, so many short ones), thirty-two rows and two
// groups beyond (every key tile is loaded half as often).  Measured, fp32, sixteen against thirty-two rows, us:
//   CTAs of sixteen rows per multiprocessor     forward          query side       key side (its own count)
//   0.9  (B 1 H 4 Hkv 2, 24 x 22, D 64)         21.4 / 35.3      40.8 / 63.0      49.2 / 88.3  (0.4)
//   3.6  (B 2 H 8 Hkv 4, 24 x 22, D 64)         55.9 / 55.0      120 / 114        86.0 / 90.1  (1.8)
//   6.9  (B 2 H 8 Hkv 4, 32 x 32, D 64)         128.8 / 119.6    276 / 256        170 / 199    (3.5)
//   10.4 (B 2 H 8 Hkv 8, 48 x 32, D 64)         232.5 / 200.5    504 / 465        313 / 297    (10.4)
//   10.4 (B 2 H 8 Hkv 4, 48 x 32, D 128)        369 / 355        822 / 795        466 / 488    (5.2)
//   10.4 (B 2 H 8 Hkv 4, 48 x 32, D 32)         129 / 136        409 / 254        204 / 224    (5.2)
// The three cross at different counts (the query side below three, the key side between five and ten); one line at four
// lies between them.
constexpr int kSmallWaves = 4;
bool few_rows(int64_t rows, int heads) { return (rows + 15) / 16 * heads <= (int64_t)kSmallWaves * device_sm_count(); }

template <typename Tin, int D, int WPG, int NG, int KN>
int run_fwd(const Args& a, cudaStream_t s) {
  constexpr int BM = 8 * WPG;
  const size_t smem = sizeof(float) * (fwd_fixed_floats<D, WPG, NG, KN>() + (size_t)BM * (a.T + a.C));
  int rc = set_smem(simt_fwd_kernel<Tin, D, WPG, NG, KN>, smem);
  if (rc) return rc;
  MVPA_CUDA_CHECK(launch_dependent(1, simt_fwd_kernel<Tin, D, WPG, NG, KN>, dim3((a.q_tn * a.C + BM - 1) / BM, a.B * a.H), 32 * WPG * NG,
                                   smem, s, a));
  count_launch();
  MVPA_CUDA_CHECK(cudaGetLastError());
  return MVPA_OK;
}

template <typename Tin, int D>
int launch_fwd(const Args& a, cudaStream_t s) {
  constexpr int KN = D == 128 ? 32 : 64;
  // the documented limit on the time and channel slots
  const size_t limit = sizeof(float) * ((size_t)32 * (D + 4) + 2 * 64 * (D + 4) + 32 * 65 + (size_t)32 * (a.T + a.C) + 3 * 32);
  if (limit > 227 * 1024) {
    set_error("fp32 path: T + C = %d needs %zu bytes of shared memory (max 232448)", a.T + a.C, limit);
    return MVPA_ERR_UNSUPPORTED;
  }
  const size_t tc = (size_t)a.T + a.C;
  if (few_rows((int64_t)a.q_tn * a.C, a.B * a.H)) {
    if (fwd_fixed_floats<D, 2, 4, KN>() + 16 * tc <= kMaxSmemFloats) return run_fwd<Tin, D, 2, 4, KN>(a, s);
  } else if (fwd_fixed_floats<D, 4, 2, KN>() + 32 * tc <= kMaxSmemFloats) {
    return run_fwd<Tin, D, 4, 2, KN>(a, s);
  }
  static_assert(fwd_fixed_floats<D, 2, 2, KN>() + 16 * ((kMaxSmemFloats - 32 * (D + 4)) / 32 - 4 * (D + 4) - 67) <= kMaxSmemFloats,
                "whatever the limit admits fits");
  return run_fwd<Tin, D, 2, 2, KN>(a, s);
}

template <typename Tin, int D, int WPG, int NG, int KN, bool INS>
int run_dq(const BwdArgs& b, size_t smem_floats, cudaStream_t s) {
  constexpr int BM = 8 * WPG;
  int rc = set_smem(simt_dq_kernel<Tin, D, WPG, NG, KN, INS>, smem_floats * sizeof(float));
  if (rc) return rc;
  MVPA_CUDA_CHECK(launch_dependent(1, simt_dq_kernel<Tin, D, WPG, NG, KN, INS>, dim3((b.a.N + BM - 1) / BM, b.a.B * b.a.H),
                                   32 * WPG * NG, smem_floats * sizeof(float), s, b));
  count_launch();
  MVPA_CUDA_CHECK(cudaGetLastError());
  return MVPA_OK;
}

template <typename Tin, int D, int WPG, int NG, int KN>
int run_dkv(const BwdArgs& b, cudaStream_t s) {
  constexpr int BM = 8 * WPG;
  constexpr size_t smem = dkv_fixed_floats<D, WPG, NG, KN>() * sizeof(float);
  static_assert(smem <= 232448, "shared memory budget");
  int rc = set_smem(simt_dkv_kernel<Tin, D, WPG, NG, KN>, smem);
  if (rc) return rc;
  // Few CTAs whose groups have more than one item each: a cluster of two CTAs shares the (head, query tile) items of the same
  // keys, and each adds up half of the rows out of the other's shared memory.  us at head_dim 64, alone / in pairs: 66 CTAs
  // (B 1 H 4 Hkv 2 T 24 C 22) 50.5 / 35.7, 96 CTAs 44.2 / 35.2, 132 CTAs 51.1 / 58.2 (more than one round of CTAs); clusters of four
  // at 66 CTAs 39.8; one item a group (12 x 8 tokens) 9.8 / 11.7.
  const unsigned tiles = (unsigned)((b.a.N + BM - 1) / BM), heads = (unsigned)(b.a.B * b.a.Hkv);
  const bool shared_items = b.a.g * ((b.a.N + KN - 1) / KN) > NG && 3 * (int64_t)tiles * heads <= 2 * (int64_t)device_sm_count();
  const unsigned parts = shared_items ? 2 : 1;
  MVPA_CUDA_CHECK(launch_dependent(parts, simt_dkv_kernel<Tin, D, WPG, NG, KN>, dim3(tiles, heads, parts), 32 * WPG * NG, smem, s, b));
  count_launch();
  MVPA_CUDA_CHECK(cudaGetLastError());
  return MVPA_OK;
}

template <typename Tin, int D>
int launch_bwd(const BwdArgs& b, cudaStream_t s) {
  const Args& a = b.a;
  if (b.tc_extra != nullptr) {
    // bf16 on the tensor cores: dq, dk, dv and the relative-key gradients
    if constexpr (sizeof(Tin) == 2 && D >= 64) {
      int rc = tc_bwd_q(b, b.tc_extra, s);
      if (rc) return rc;
      return tc_bwd_bias(b, b.tc_extra, s);
    }
  }
  constexpr int KN = D == 128 ? 32 : 64;
  const size_t limit = sizeof(float) * ((size_t)2 * 32 * (D + 4) + 2 * 64 * (D + 4) + 2 * 32 * 65 + (size_t)32 * (a.T + a.C) + 2 * 32 + 16 * D);
  if (limit > 227 * 1024) {
    set_error("fp32 backward: T + C = %d needs %zu bytes of shared memory", a.T + a.C, limit);
    return MVPA_ERR_UNSUPPORTED;
  }
  const size_t tc = (size_t)a.T + a.C;
  const size_t small_f = dq_fixed_floats<D, 2, 4, KN>() + 16 * 5 * tc, large_f = dq_fixed_floats<D, 4, 2, KN>() + 32 * 3 * tc;
  int rc, bm = 16;
  if (few_rows(a.N, a.B * a.H) && small_f <= kMaxSmemFloats) {
    rc = run_dq<Tin, D, 2, 4, KN, true>(b, small_f, s);
  } else if (!few_rows(a.N, a.B * a.H) && large_f <= kMaxSmemFloats) {
    rc = run_dq<Tin, D, 4, 2, KN, true>(b, large_f, s);
    bm = 32;
  } else {
    static_assert(dq_fixed_floats<D, 2, 2, 32>() + 32 * ((kMaxSmemFloats - 64 * (D + 4) - 4224 - 16 * D) / 32 - 4 * (D + 4)) <= kMaxSmemFloats,
                  "whatever the limit admits fits");
    rc = run_dq<Tin, D, 2, 2, 32, false>(b, dq_fixed_floats<D, 2, 2, 32>() + 32 * tc, s);
  }
  if (rc) return rc;
  rc = few_rows(a.N, a.B * a.Hkv) ? run_dkv<Tin, D, 2, 4, KN>(b, s) : run_dkv<Tin, D, 4, 2, KN>(b, s);
  if (rc) return rc;
  const int n_qt = (a.N + bm - 1) / bm;
  const int n_chunks = a.B * a.g * ((a.N + kDrelRows - 1) / kDrelRows);
  const int n_z = n_chunks < kDrelSplit ? n_chunks : kDrelSplit;
  {
    const size_t smem = sizeof(float) * ((size_t)kDrelRows * (kDrelSlots + 1) + kDrelRows * (D + 4));
    rc = set_smem(simt_drel_kernel<Tin, D>, smem);
    if (rc) return rc;
    const unsigned blocks = (a.T + kDrelSlots - 1) / kDrelSlots + (a.C + kDrelSlots - 1) / kDrelSlots;
    MVPA_CUDA_CHECK(launch_dependent(1, simt_drel_kernel<Tin, D>, dim3(blocks, a.Hkv, n_z), kThreads, smem, s, b));
  }
  const int64_t total = (int64_t)a.Hkv * (a.T + a.C) * D;
  const int n_red = (int)((total + kThreads - 1) / kThreads < 592 ? (total + kThreads - 1) / kThreads : 592);
  MVPA_CUDA_CHECK(launch_dependent(1, simt_final_kernel, n_red + 3 * a.Hkv, kThreads, 0, s, b, n_z, n_qt, n_red));
  count_launch(2);
  MVPA_CUDA_CHECK(cudaGetLastError());
  return MVPA_OK;
}

template <typename Tin>
int dispatch_fwd(const Args& a, cudaStream_t s) {
  switch (a.D) {
    case 16: return launch_fwd<Tin, 16>(a, s);
    case 32: return launch_fwd<Tin, 32>(a, s);
    case 64: return launch_fwd<Tin, 64>(a, s);
    case 128: return launch_fwd<Tin, 128>(a, s);
  }
  return MVPA_ERR_SHAPE;
}

template <typename Tin>
int dispatch_bwd(const BwdArgs& b, cudaStream_t s) {
  switch (b.a.D) {
    case 16: return launch_bwd<Tin, 16>(b, s);
    case 32: return launch_bwd<Tin, 32>(b, s);
    case 64: return launch_bwd<Tin, 64>(b, s);
    case 128: return launch_bwd<Tin, 128>(b, s);
  }
  return MVPA_ERR_SHAPE;
}

}  // namespace

int simt_fwd(const Args& a, int dtype, cudaStream_t s) {
  return dtype == MVPA_F32 ? dispatch_fwd<float>(a, s)
         : dtype == MVPA_F16 ? dispatch_fwd<__half>(a, s) : dispatch_fwd<__nv_bfloat16>(a, s);
}

int simt_bwd(const BwdArgs& b, int dtype, cudaStream_t s) {
  return dtype == MVPA_F32 ? dispatch_bwd<float>(b, s)
         : dtype == MVPA_F16 ? dispatch_bwd<__half>(b, s) : dispatch_bwd<__nv_bfloat16>(b, s);
}

namespace {
// bf16 problems the tensor-core backward takes need only delta from this file's areas; everything else lives in tc_extra.
bool tc_path(int dtype, int D, int C, int T) {
  Args a{};
  a.D = D; a.C = C; a.T = T;
  return dtype == MVPA_BF16 && tc_bwd_q_supported(a);
}
// delta, in front of the tensor-core kernels' own workspace
size_t tc_head_floats(size_t rows) { return (rows + 63) & ~(size_t)63; }
}  // namespace

size_t simt_bwd_workspace_floats(const mvpa_problem* p) {
  const size_t BH = (size_t)p->B * p->H, N = (size_t)p->T * p->C;
  if (tc_path(p->dtype, p->D, p->C, p->T)) {
    return tc_head_floats(BH * N) + tc_bwd_q_workspace_floats(p);
  }
  const size_t n_qt = (N + kMinRows - 1) / kMinRows;  // at most
  size_t n = 2 * BH * N * (p->T + p->C) + BH * N + BH * n_qt * 3 * p->D;
  n = ((n + 3) & ~(size_t)3) + (size_t)kDrelSplit * p->Hkv * (p->T + p->C) * p->D;
  return (n + 63) & ~(size_t)63;
}

const int* bwd_status_word(const mvpa_problem* p, const void* workspace) {
  if (!tc_path(p->dtype, p->D, p->C, p->T)) return nullptr;  // the CUDA-core kernels have no device-side waits
  const size_t BH = (size_t)p->B * p->H, N = (size_t)p->T * p->C;
  return reinterpret_cast<const int*>(static_cast<const float*>(workspace) + tc_head_floats(BH * N) +
                                      tc_bwd_status_offset_floats(p));
}

void simt_bwd_carve(BwdArgs& b, float* ws, int dtype) {
  const Args& a = b.a;
  const size_t BH = (size_t)a.B * a.H, N = a.N;
  if (tc_path(dtype, a.D, a.C, a.T)) {
    b.tbg = b.cbg = b.dtbg = b.dcbg = b.partial = b.drel_part = nullptr;
    b.delta = ws;
    b.tc_extra = ws + tc_head_floats(BH * N);
    return;
  }
  const size_t n_qt = (N + kMinRows - 1) / kMinRows;  // at most
  b.tbg = ws;
  b.cbg = b.tbg + BH * N * a.T;
  b.dtbg = b.cbg + BH * N * a.C;
  b.dcbg = b.dtbg + BH * N * a.T;
  b.delta = b.dcbg + BH * N * a.C;
  b.partial = b.delta + BH * N;
  const size_t used = 2 * BH * N * (a.T + a.C) + BH * N + BH * n_qt * 3 * a.D;
  b.drel_part = ws + ((used + 3) & ~(size_t)3);  // stored in 16-byte pieces
  b.tc_extra = nullptr;
}

}  // namespace mvpa
