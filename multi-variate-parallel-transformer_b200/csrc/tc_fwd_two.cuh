// Flash-MVPA forward for bf16, head_dim 64 and at most 64 channel slots, two CTAs per multiprocessor (included by
// mvpa_tc_fwd.cu, whose tensor maps, argument record and small helpers it uses).
//
// One CTA owns 128 query rows of one (batch, head) as in tc_fwd_kernel, but with ONE softmax warpgroup (thread = TMEM lane
// = query row, all 128 key columns), half of the tensor memory and half of the shared memory, so that two CTAs are resident:
// the prologue, the softmax chains and the epilogue of one run under the products of the other.  At these sizes a CTA
// spends more than half of its time in such parts (a row's relative products, their gather, accumulator merge, output),
// and tc_fwd_kernel has nothing to put under them.
//
//   warps 0-3  softmax;  warp 4  TMA producer (one lane);  warp 5  MMA issuer (convergent, elected lane);  6, 7 donate registers
//
// Tiles are visited light-first: every light tile's score is its temporal score alone, so its probabilities need one
// bf16 value per (row, key time step).  These are formed once, in the prologue, against the maximum over all light tiles,
// and wait packed in tensor memory; a light tile costs the row's packed multiplies and nothing else, and its sums
// need no rescaling.  The dense tiles follow with the usual running maximum.
//
// TMEM columns (256): [0,128) S / P (light tiles: two P buffers of 64), [128,192) O, [192,256) X.  X holds the packed
// light factors of key step t at column t / 2; in a CTA without light tiles, the fp32 temporal scores of the last 64 slots.
// The prologue passes the raw temporal products through S and the raw channel products through O.
// Shared memory: Q', a ring of five 16 KB K/V slots (the prologue borrows three), and the fp32 temporal scores of the
// dense tiles' key steps: kTdSteps of them beside the ring; in a CTA without light tiles the slots before the last 64 take
// two ring slots for good.
#pragma once

namespace mvpa {
namespace {
namespace two {

constexpr int kThreads2 = 256;
constexpr int kTmemCols2 = 256;
constexpr uint32_t kS = 0, kO = 128, kX = 192;
constexpr int kTile = 16384;       // 128 rows x 64 bf16: a Q tile, a ring slot
constexpr int kSlots = 5, kEarly = 2;
constexpr int kTdSteps = 16;       // key steps of a CTA's dense tiles when it has light tiles as well
enum Bar2 { kProFull = 0, kProMma, kProDone, kSFull, kPFull, kAllDone, kPl, kPl1, kSlotFull2, kSlotFree2 = kSlotFull2 + kSlots, kBars2 = kSlotFree2 + kSlots };
constexpr int kSmemRing = kTile, kSmemTd = kSmemRing + kSlots * kTile, kSmemTail = kSmemTd + kTdSteps * 512;
constexpr int kSmemBytes = kSmemTail + (64 + 256) * 4 + kBars2 * 8 + 16 + 1024;
static_assert(2 * (kSmemBytes + 1024) <= 233472, "two CTAs per multiprocessor");

__device__ __forceinline__ void bar128() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

template <int CP>
__global__ void __launch_bounds__(kThreads2, 2)
tc_fwd_two_kernel(const __grid_constant__ TcMaps maps, const TcArgs p) {
  constexpr int D = 64, TPB = 128 / CP, KSTEPS = D / 16, LDP = CP + 2;
  static_assert(CP == 32 || CP == 64, "CP in {32,64}");

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* ring = smem + kSmemRing;
  uint8_t* sR = ring + kEarly * kTile;                   // r_time rows 0..127 (rows >= T are zero)
  uint8_t* sC = sR + kTile;                              // r_chan rows 0..CP-1
  float* scratch = reinterpret_cast<float*>(sR);         // [128][LDP], once sR / sC are dead
  float* s_far = reinterpret_cast<float*>(ring + 3 * kTile);  // [64 slots][128 rows]: CTAs without light tiles, T > 64
  float* s_td = reinterpret_cast<float*>(smem + kSmemTd);     // [kTdSteps][128 rows]
  float* s_bias = reinterpret_cast<float*>(smem + kSmemTail);  // u as fp32
  float* s_vr = s_bias + 64;
  float* s_zc = s_vr + 128;
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_zc + 128);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kBars2);
  int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);
  int* s_giveup = s_abort + 1;
  uint64_t* slot_full = bars + kSlotFull2;
  uint64_t* slot_free = bars + kSlotFree2;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int BH = p.B * p.H;
  int I_loc, bh;  // latest (heaviest) query tiles first, over all heads or inside one kv head
  if (p.kv_major) {
    const int per = p.q_tiles * p.g, grp = (int)(blockIdx.x / per), r = (int)(blockIdx.x % per);
    I_loc = p.q_tiles - 1 - r / p.g;
    bh = grp * p.g + r % p.g;  // grp = b * Hkv + hk
  } else {
    I_loc = p.q_tiles - 1 - (int)(blockIdx.x / BH);
    bh = blockIdx.x % BH;
  }
  const int I = p.q_t0 / TPB + I_loc;
  const int b = bh / p.H, h = bh % p.H, hk = h / p.g;
  const int n_light = light_tiles(I, TPB, p.window, p.n_qt), n_dense = I + 1 - n_light;
  const int T = p.T, C = p.C;
  const int ns = n_light == 0 && T > 64 ? 3 : kSlots;  // ring slots in use
  struct Cursor {  // walks the ring in load order: slot and the parity of its use
    uint32_t sl, par;
    __device__ __forceinline__ void next(int n) {
      if (++sl == (uint32_t)n) { sl = 0; par ^= 1; }
    }
  };

  if (tid == 0) {
    *s_giveup = 0;
    for (int i = 0; i < kBars2; ++i)
      mbar_init(&bars[i], i == kProDone || i == kPFull || i == kPl || i == kPl1 ? 128 : 1);
    mbar_fence_init();
  }
  if (warp == 5) {
    tmem_alloc(tmem_slot, kTmemCols2);
    tmem_relinquish();
  }
  griddep_wait();  // nothing above reads memory; the status words and constants come from the pre-kernel
  if (tid == 64) *s_abort = *p.status;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (*s_abort != 0) {  // do nothing, but give the columns back
    if (warp == 5) tmem_dealloc(tmem, kTmemCols2);
    return;
  }
  // (208 and 40 registers a thread: 31744 of the 32768 the CTA was launched with)
  if (warp >= 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
  if (warp == 4) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      prefetch_tensormap(&maps.q);
      prefetch_tensormap(&maps.k);
      prefetch_tensormap(&maps.v);
      mbar_arrive_expect_tx(&bars[kProFull], 2 * kTile + CP * 128);
      tma_load_5d(sQ, &maps.q, &bars[kProFull], 0, 0, I_loc * TPB, h, b);
      tma_load_3d(sR, &maps.rt, &bars[kProFull], 0, 0, hk);
      tma_load_3d(sC, &maps.rc, &bars[kProFull], 0, 0, hk);
      bool ok = true;
      Cursor at{0, 1};  // (parity of the slot's previous release)
      int q = 0;
      auto load_slot = [&](const CUtensorMap* map, int J) {
        if (q == kEarly) ok = mbar_wait(&bars[kProDone], 0, p.status, 10);  // borrowed slots are back
        if (ok && q >= ns) ok = mbar_wait(&slot_free[at.sl], at.par, p.status, 11);
        if (!ok) return;
        mbar_arrive_expect_tx(&slot_full[at.sl], kTile);
        tma_load_5d(ring + at.sl * kTile, map, &slot_full[at.sl], 0, 0, J * TPB, hk, b);
        at.next(ns);
        ++q;
      };
      for (int J = 0; ok && J < n_light + n_dense; ++J) {
        if (J >= n_light) load_slot(&maps.k, J);
        if (ok) load_slot(&maps.v, J);
      }
    }
  } else if (warp == 5) {
    // ------------------------------- MMA issuer -------------------------------
    constexpr uint32_t kFull = 0xffffffffu;
    const uint32_t el = elect_one();
    const uint32_t tm = __shfl_sync(kFull, tmem, 0);
    constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, 0);
    constexpr uint32_t idesc_c = make_idesc_bf16(128, CP, 0);
    constexpr uint32_t idesc_o = make_idesc_bf16(128, D, 1);
    bool ok = __all_sync(kFull, mbar_wait(&bars[kProFull], 0, p.status, 20));
    const DescHalves dq = make_desc_halves_sw128(smem_u32(sQ), 16, 1024);
    if (ok) {
      tc_fence_after();
      const DescHalves dr = make_desc_halves_sw128(smem_u32(sR), 16, 1024);
      const DescHalves dc = make_desc_halves_sw128(smem_u32(sC), 16, 1024);
#pragma unroll
      for (int kk = 0; kk < KSTEPS; ++kk) mma_ss_w(el, tm + kO, dq, kk * 32, dc, kk * 32, idesc_c, kk > 0);
#pragma unroll
      for (int kk = 0; kk < KSTEPS; ++kk) mma_ss_w(el, tm + kS, dq, kk * 32, dr, kk * 32, idesc_s, kk > 0);
      mma_commit_w(el, smem_u32(&bars[kProMma]));
      ok = __all_sync(kFull, mbar_wait(&bars[kProDone], 0, p.status, 21));  // Q rewritten as (q+u) c2; S and O free
    }
    const DescHalves dk0 = make_desc_halves_sw128(smem_u32(ring), 16, 1024);
    const DescHalves dv0 = make_desc_halves_sw128(smem_u32(ring), kTile, 1024);
    const uint32_t a_full = smem_u32(slot_full), a_free = smem_u32(slot_free);
    const uint32_t a_sfull = smem_u32(&bars[kSFull]), a_pfull = smem_u32(&bars[kPFull]), a_pl = smem_u32(&bars[kPl]);
    Cursor at{0, 0};
    // O += P V of the tile whose V is next in the ring; P at TMEM column `a0`, 64 columns
    auto issue_pv = [&](uint32_t a0, uint32_t acc) {
      const uint32_t b_lo = dv0.lo + at.sl * (kTile >> 4);
      mma_ts_x4_w(el, tm + kO, a0, b_lo, dv0.hi, 2048 >> 4, idesc_o, acc);
      mma_ts_x4_w(el, tm + kO, a0 + 32, b_lo + 4 * (2048 >> 4), dv0.hi, 2048 >> 4, idesc_o, 1u);
      mma_commit_w(el, a_free + 8 * at.sl);
      at.next(ns);
    };
    // ---- light tiles ----
    for (int l = 0; ok && l < n_light; ++l) {
      ok = __all_sync(kFull, mbar_wait_a(a_full + 8 * at.sl, at.par, p.status, 24));
      if (ok) ok = __all_sync(kFull, mbar_wait_a(a_pl + 8 * (l & 1), (l >> 1) & 1, p.status, 23));
      if (!ok) break;
      tc_fence_after();
      issue_pv(tm + kS + 64 * (l & 1), (uint32_t)(l > 0));
    }
    // ---- dense tiles: S of the next tile goes out behind the PV product that reads the columns it overwrites ----
    for (int e = 0; ok && e < n_dense; ++e) {
      ok = __all_sync(kFull, mbar_wait_a(a_full + 8 * at.sl, at.par, p.status, 22));
      if (!ok) break;
      tc_fence_after();
      DescHalves dk = dk0;
      dk.lo += at.sl * (kTile >> 4);
#pragma unroll
      for (int kk = 0; kk < KSTEPS; ++kk) mma_ss_w(el, tm + kS, dq, kk * 32, dk, kk * 32, idesc_s, kk > 0);
      mma_commit_w(el, a_sfull);
      mma_commit_w(el, a_free + 8 * at.sl);
      at.next(ns);
      ok = __all_sync(kFull, mbar_wait_a(a_full + 8 * at.sl, at.par, p.status, 24));
      if (ok) ok = __all_sync(kFull, mbar_wait_a(a_pfull, e & 1, p.status, 23));
      if (!ok) break;
      tc_fence_after();
      issue_pv(tm + kS, (uint32_t)(n_light > 0 || e > 0));
    }
    mma_commit_w(el, smem_u32(&bars[kAllDone]));
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    // ------------------------------ softmax warps ------------------------------
    const int row = tid;  // query row of the tile == TMEM lane
    const int ti_loc = row / CP, c_i = row % CP;
    const int ti_abs = I * TPB + ti_loc;
    const bool row_valid = c_i < C && ti_abs < p.q_t0 + p.q_tn;
    const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
    if (row < D) s_bias[row] = __bfloat162float(p.u[hk * D + row]);
    s_vr[row] = p.relc[hk * 256 + row];
    s_zc[row] = p.relc[hk * 256 + 128 + row];
    bar128();
    bool ok = warp_wait(&bars[kProFull], 0, p.status, 30);
    if (ok) ok = warp_wait(&bars[kProMma], 0, p.status, 31);
    // Channel scores of the row, c2 (q.r_chan[j] + z.r_chan[j]), into this thread's own row of the scratch
    // (the relative-key tiles there were only read by the two products).
    if (ok) {
      tc_fence_after();
#pragma unroll
      for (int ci = 0; ci < CP / 32; ++ci) {
        uint32_t v[32];
        tmem_ld32(lane_base + kO + ci * 32, v);
        tmem_ld_wait();
#pragma unroll
        for (int jj = 0; jj < 32; jj += 2) {
          const float2 zc = *reinterpret_cast<const float2*>(s_zc + ci * 32 + jj);
          *reinterpret_cast<float2*>(scratch + row * LDP + ci * 32 + jj) =
              make_float2(p.c2 * (__uint_as_float(v[jj]) + zc.x), p.c2 * (__uint_as_float(v[jj + 1]) + zc.y));
        }
      }
    }
    // Gathered by |c_i - c_k|: cbf = cb - max (fp32, log2 domain).  Slot C-1-|c_i - c_k| runs up through the row for
    // c_k <= c_i and down for c_k > c_i: two base pointers with constant offsets (rows padded by two floats: no bank
    // conflicts on either diagonal; positions of channels that do not exist may lie outside the row, their values are dropped).
    float cbf[CP];
    float mc;
    {
      const float* up = scratch + row * LDP + (C - 1 - c_i);
      const float* down = scratch + row * LDP + (C - 1 + c_i);
      const int climit = c_i < C ? C : 0;
      float mx = -INFINITY;
#pragma unroll
      for (int k = 0; k < CP; ++k) {
        const float val = k <= c_i ? up[k] : down[-k];
        cbf[k] = ok && k < climit ? val : -INFINITY;
        mx = fmaxf(mx, cbf[k]);
      }
      mc = mx == -INFINITY ? 0.f : mx;
#pragma unroll
      for (int k = 0; k < CP; ++k) cbf[k] -= mc;
    }
    if (ok) {  // Q' = (q+u) c2 in place (`attentions/attn.py:180-183`)
      const float4* u4 = reinterpret_cast<const float4*>(s_bias);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const uint32_t off = row * 128 + ((c ^ (row & 7)) << 4);
        const uint4 raw = *reinterpret_cast<const uint4*>(sQ + off);
        const float4 b0 = u4[c * 2], b1 = u4[c * 2 + 1];
        uint4 out;
        out.x = pack_bf16((__uint_as_float(raw.x << 16) + b0.x) * p.c2, (__uint_as_float(raw.x & 0xffff0000u) + b0.y) * p.c2);
        out.y = pack_bf16((__uint_as_float(raw.y << 16) + b0.z) * p.c2, (__uint_as_float(raw.y & 0xffff0000u) + b0.w) * p.c2);
        out.z = pack_bf16((__uint_as_float(raw.z << 16) + b1.x) * p.c2, (__uint_as_float(raw.z & 0xffff0000u) + b1.y) * p.c2);
        out.w = pack_bf16((__uint_as_float(raw.w << 16) + b1.z) * p.c2, (__uint_as_float(raw.w & 0xffff0000u) + b1.w) * p.c2);
        *reinterpret_cast<uint4*>(sQ + off) = out;
      }
      fence_proxy_async_smem();
    }
    // ---- temporal scores, c2 (q.r_time[j] + vt.r_time[j]) + channel maximum, out of the S columns ----
    // Key step t of this row is column col0 + t (uniform in a warp: its rows share a time step).  Short loops: they run
    // once per CTA.
    const int col0 = T - 1 - ti_abs, light_steps = n_light * TPB, near0 = max(T - 64, 0);
    auto score = [&](uint32_t raw, int col) { return p.c2 * (__uint_as_float(raw) + s_vr[col]) + mc; };
    float m_used = -INFINITY;
    float l_sum[2] = {0.f, 0.f};  // light tiles by half, dense tiles by parity (as in tc_fwd_kernel, whose warpgroups hold one each)
    if (n_light == 0) {
      // every key step may be needed in fp32: the last 64 slots go to X, those before them to shared memory
      // (once all threads are done with the scratch there)
      bar128();
#pragma unroll 1
      for (int c = 0; c < 64; c += 8) {
        uint32_t v[8];
        tmem_ld8(lane_base + kS + near0 + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) v[jj] = __float_as_uint(score(v[jj], near0 + c + jj));
        tmem_st8(lane_base + kX + c, v);
      }
#pragma unroll 1
      for (int c = 0; c < near0; c += 8) {
        uint32_t v[8];
        tmem_ld8(lane_base + kS + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) s_far[(c + jj) * 128 + row] = score(v[jj], c + jj);
      }
    } else {
#pragma unroll
      for (int c = 0; c < kTdSteps; c += 8) {
        uint32_t v[8];
        const int j0 = col0 + light_steps + c;
        tmem_ld8(lane_base + kS + j0, v);
        tmem_ld_wait();
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) s_td[(c + jj) * 128 + row] = score(v[jj], j0 + jj);  // (t_k > t_i: not used)
      }
      m_used = kLowest;
#pragma unroll 1
      for (int c = 0; c < light_steps; c += 16) {
        uint32_t v[2][8];
        tmem_ld8(lane_base + kS + col0 + c, v[0]);
        tmem_ld8(lane_base + kS + col0 + c + 8, v[1]);
        tmem_ld_wait();
#pragma unroll
        for (int jj = 0; jj < 16; ++jj)
          if (c + jj < light_steps) m_used = fmaxf(m_used, score(v[jj / 8][jj % 8], col0 + c + jj));
      }
#pragma unroll 1
      for (int c = 0; c < light_steps; c += 16) {
        uint32_t v[2][8], w[8];
        tmem_ld8(lane_base + kS + col0 + c, v[0]);
        tmem_ld8(lane_base + kS + col0 + c + 8, v[1]);
        tmem_ld_wait();
#pragma unroll
        for (int jj = 0; jj < 16; jj += 2)
          w[jj / 2] = pack_bf16(ex2(score(v[jj / 8][jj % 8], col0 + c + jj) - m_used),
                                ex2(score(v[jj / 8][jj % 8 + 1], col0 + c + jj + 1) - m_used));
        tmem_st8(lane_base + kX + c / 2, w);
      }
    }
    tmem_st_wait();
    tc_fence_before();
    mbar_arrive(&bars[kProDone]);  // borrowed ring slots, S, O and the rewritten Q are ready

    // ------------------------------ light tiles ------------------------------
    // P[i,k] = a_i[t_k] bc_i[c_k], packed bf16 products of the factors in X and the row's channel vector; two buffers.
    if (ok && n_light > 0) {
      Cursor pv{0, 0};  // ring position of the V whose product frees the buffer written next (two tiles back)
      uint32_t bc[CP / 2];  // exp2(channel score - its maximum), bf16 pairs
      float sum_bc = 0.f;
#pragma unroll
      for (int k2 = 0; k2 < CP / 2; ++k2) {
        bc[k2] = pack_bf16(ex2(cbf[2 * k2]), ex2(cbf[2 * k2 + 1]));
        sum_bc += __uint_as_float(bc[k2] << 16) + __uint_as_float(bc[k2] & 0xffff0000u);
      }
      uint32_t aw[TPB / 2];  // the tile's factors
      auto fetch = [&](int l) {
#pragma unroll
        for (int j = 0; j < TPB / 2; ++j) tmem_ld1(lane_base + kX + l * (TPB / 2) + j, aw[j]);
      };
      fetch(0);
      for (int l = 0; l < n_light; ++l) {
        uint32_t p0[32], p1[32];
        tmem_ld_wait();
#pragma unroll
        for (int tt = 0; tt < TPB; ++tt) {
          const uint32_t a2 = __byte_perm(aw[tt / 2], 0, tt & 1 ? 0x3232 : 0x1010);
          l_sum[tt / (TPB / 2)] += __uint_as_float(a2 & 0xffff0000u) * sum_bc;
#pragma unroll
          for (int k2 = 0; k2 < CP / 2; ++k2) {
            const int idx = tt * (CP / 2) + k2;
            if (idx < 32) p0[idx] = hmul2_bf16(a2, bc[k2]);
            else p1[idx - 32] = hmul2_bf16(a2, bc[k2]);
          }
        }
        if (l + 1 < n_light) fetch(l + 1);
        if (l >= 2) {
          ok = warp_wait(&slot_free[pv.sl], pv.par, p.status, 35);
          if (!ok) break;
          pv.next(ns);
          tc_fence_after();
        }
        const uint32_t addr = lane_base + kS + 64 * (l & 1);
        tmem_st32(addr, p0);
        tmem_st32(addr + 32, p1);
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive(&bars[kPl + (l & 1)]);
      }
    }

    // ------------------------------ dense tiles ------------------------------
    const uint32_t s_addr = lane_base + kS;
    for (int e = 0; ok && e < n_dense; ++e) {
      const int J = n_light + e;
      DenseTile<CP> t;
#pragma unroll
      for (int tt = 0; tt < TPB; ++tt) {
        const int tk_abs = J * TPB + tt, dt = ti_abs - tk_abs;
        t.valid[tt] = dt >= 0 && tk_abs < T;
        t.wmul[tt] = (p.window > 0 && dt > p.window && ti_abs != T - 1) ? 0.f : 1.f;
        const int slot = T - 1 - min(max(dt, 0), T - 1);  // (uniform in a warp)
        if (n_light > 0) {
          t.tb[tt] = s_td[(e * TPB + tt) * 128 + row];
        } else if (slot >= near0) {
          uint32_t raw;
          tmem_ld1(lane_base + kX + slot - near0, raw);
          tmem_ld_wait();
          t.tb[tt] = __uint_as_float(raw);
        } else {
          t.tb[tt] = s_far[slot * 128 + row];
        }
      }
      ok = warp_wait(&bars[kSFull], e & 1, p.status, 32);
      if (!ok) break;
      tc_fence_after();
      uint32_t va[32];
      const float m_tile = dense_max<CP>(s_addr, t, cbf, va);
      if (e == 0 && n_light == 0) {
        m_used = (m_tile == -INFINITY) ? 0.f : m_tile;
      } else {
        // O and l follow the maximum only when it moved by more than 2^8 (every PV product so far is complete: the
        // score product that has just been waited for was issued behind them)
        const bool need = m_tile > m_used + kRescaleThreshold;
        if (__any_sync(0xffffffffu, need)) {
          const float alpha = need ? ex2(m_used - m_tile) : 1.f;
          rescale_columns(lane_base + kO, D, alpha);
          l_sum[0] *= alpha;
          l_sum[1] *= alpha;
          if (need) m_used = m_tile;
        }
      }
      const float psum = dense_exp<CP>(s_addr, t, cbf, m_used, va);
      if (e & 1) l_sum[1] += psum;
      else l_sum[0] += psum;
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&bars[kPFull]);
    }
    // ------------------------------- epilogue ---------------------------------
    if (ok) ok = warp_wait(&bars[kAllDone], 0, p.status, 34);
    if (ok) {
      tc_fence_after();
      const float l = l_sum[0] + l_sum[1], inv = 1.f / l;
      // O / l as bf16 into the Q tile's place (laid out like it), then one TMA store; rows and channels outside the
      // tensor are not written.
      uint32_t va[32], vb[32];
      tmem_ld32(lane_base + kO, va);
      tmem_ld32(lane_base + kO + 32, vb);
      tmem_ld_wait();
      auto put = [&](const uint32_t (&v)[32], int c0) {
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            w[j] = pack_bf16(__uint_as_float(v[q4 * 8 + 2 * j]) * inv, __uint_as_float(v[q4 * 8 + 2 * j + 1]) * inv);
          *reinterpret_cast<uint4*>(sQ + row * 128 + (((c0 + q4) ^ (row & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      };
      put(va, 0);
      put(vb, 4);
      fence_proxy_async_smem();
      if (row_valid && p.lse != nullptr)
        p.lse[(int64_t)bh * p.q_tn * C + (int64_t)(ti_abs - p.q_t0) * C + c_i] = m_used + log2f(l);
    }
    if (!ok) *s_giveup = 1;
    bar128();
    if (*s_giveup == 0 && tid == 0) {
      tma_store_5d(&maps.o, sQ, 0, 0, I_loc * TPB, h, b);
      tma_store_commit();
      tma_store_wait_all();
    }
    tc_fence_before();
  }
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols2);
  }
}

// Whether a call takes this kernel.
//   * Enough CTAs: a single CTA is faster with two softmax warpgroups on a multiprocessor of its own, so the longest one (the
//     last query tile, n_qt dense tiles: 6.5 + 1.5 n_qt us here) has to be shorter than the whole call in the other kernel.
//     That is where the CTAs outnumber the multiprocessors 1.15 + n_qt / 20 times.  Measured, us, this kernel / the other as it
//     is now (calls back to back, pre-kernel included; 64 channels, 12 heads):  n_qt 2: 144 CTAs 12.4 / 9.9, 168 12.5 / 17.1, 192
//     12.7 / 17.6;  6: 144 17.1 / 13.6, 216 18.3 / 20.5;  13: 156 26.2 / 21.7, 312 29.4 / 33.3;  32: 384 59.1 / 48.6, 768 69.0 / 88.1;
//     64: 768 110 / 114, 1536 171 / 216.  Large calls: 4 x 64 x 64 tokens, 16 heads 170 / 228, 8 x 128 x 64, 12 heads 664 / 841,
//     8 x 128 x 32, 16 heads 302 / 407.  (At 32 slots a CTA's tiles are the shorter ones and the line lies a little early: 1 x 128 x 32,
//     16 heads, 512 CTAs 62 / 56; 2 x 40 x 22, 12 heads, 240 CTAs 24 / 22 stays with the other.)
//     Large calls that the other kernel keeps for their window: 4 x 64 x 64 tokens, window 15 248, 40 302; 8 x 128 x 64, 12 heads, window 15
//     925, 40 1182; 8 x 128 x 32, window 13 423, 40 499.
//   * A content window whose dense key steps fit s_td (every shipped window, 10, does; a window past the last key step, or
//     none, leaves no light tiles and needs no s_td).
inline bool applies(int window, int CP, int n_qt, unsigned grid) {
  const int TPB = 128 / CP;
  const bool any_light = window > 0 && n_qt >= 2 && (n_qt - 2) * TPB - TPB - window >= 0;
  return 20 * (int64_t)grid > (int64_t)device_sm_count() * (23 + n_qt) &&
         (!any_light || ((window + TPB - 1) / TPB + 1) * TPB <= kTdSteps);
}

}  // namespace two
}  // namespace
}  // namespace mvpa
