// Resident 2D integration: one thread-block cluster per sample advances every SETDRK4 step and
// stage in one launch, with the sample's state, running sums, stage fields and products in the
// cluster's shared memory. The column and row passes (fsm_plane_reg.cuh) exchange their fields
// through global memory and one launch each; here the exchange is a store into the owner's shared
// memory (distributed shared memory) and a cluster barrier. Same arithmetic as the passes,
// operation by operation, so that a sample's result does not depend on which of the two ran it.
//
// Split. Of the H = NY/2 + 1 columns of the half spectrum a CTA owns ka of the HK kept ones (the
// 2/3 rule's prefix, which need the inverse transforms) and kb of the rest, and it owns NX / CL
// rows (CL: cluster size). Per stage:
//   row phase: c2r of the CTA's rows of the stage fields (MID, in its shared memory), products,
//     r2c, each product value stored to the CTA that owns its column (PROD there);
//   column phase: x transform of the CTA's columns of PROD, stage update, next-stage fields, their
//     inverse x transforms, each value stored to the CTA that owns its row (MID there).
// A group of T lanes keeps a column (row) in registers from its first transform to its last, so a
// phase needs no CTA-wide barrier. FS groups share a column's inverse transforms where columns are
// few (each repeats the forward transform and the update; the first one writes the state).
//
// Bound: the latency of a stage's chain (three to six transforms, two cluster barriers of 500-800
// cycles) at one to eight warps per SM, then instruction issue. 2D Burgers 64^2 x 1: 83 -> 12.7 us
// per step (8 launches a step of 2 and 1 CTAs before); vorticity 64^2 x 4: 65 -> 11.6; velocity
// Navier-Stokes 128 x 256 x 9: 170 -> 51; Burgers 128^2 x 16: 150 -> 33.
#pragma once

#include "fsm_plane_reg.cuh"

namespace fsm {

struct ResArgs {
  StepArgs a;
  int ka, kb;  // kept / other columns per CTA
  int pc;      // PROD row pitch (>= ka + kb, odd)
  int fs;      // groups per column
  int rpc;     // rows per CTA (even; the last CTAs may have fewer)
  int tables;  // every coefficient table in shared memory; else those of stage 0 alone (E - 1, E2 - 1, c4) in global memory
};

constexpr int kResThreads = 256;

template <int NX, int NY, int KIND>
struct ResCfg {
  static constexpr int C = RegKind<KIND, 2>::C;
  static constexpr int NP = C;
  static constexpr int NM = 4;
  static constexpr int TX = RegShape<NX>::T, EX = RegShape<NX>::E;
  static constexpr int TY = RegShape<NY>::T, EY = RegShape<NY>::E;
  static constexpr int H = NY / 2 + 1, HK = NY / 3 + 1;
  // state column pitch: the groups of a half-warp on distinct banks (one group when T is 16)
  static constexpr int SP = NX + (TX < 16 ? TX : 0);
  static constexpr int WSX = (32 / TX) * reg_scratch<NX>(), WSY = (32 / TY) * reg_scratch<NY>();
  static constexpr int WS = WSX > WSY ? WSX : WSY;  // transform scratch per warp
  // shared memory of a CTA (float2 units) for rpc rows per CTA
  static size_t smem(int rpc, int ka, int kb, int pc, int fs, int tch, bool tables, int threads) {
    const int rp = rpc | 1;
    size_t w = (size_t)NX + NY;                        // transform twiddles
    w += (size_t)NM * HK * rp;                         // MID
    w += (size_t)NP * NX * pc;                         // PROD
    w += (size_t)(fs > 1 ? 4 : 3) * C * (ka + kb) * SP;  // u, q, acc (and B when groups share columns)
    w += (size_t)(threads / 32) * WS;
    // coefficient tables: (c1, c5), then (c6, c4), E2 - 1 and E - 1, or c6 alone (floats; SP is even)
    w += (size_t)tch * (ka + kb) * SP * (tables ? 8 : 3) / 2;
    if (KIND == FSM_NL_LERAY) w += (size_t)(ka + kb) * SP / 2;  // 1 / lap (floats; SP is even)
    w += NX + (H + 1) / 2;                             // kx, row mask, ky (floats)
    return w * sizeof(float2) + (size_t)(H + 1) * sizeof(uint16_t);
  }
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Store v at the address `local` has in the shared memory of CTA `rank` of the cluster.
__device__ __forceinline__ void st_cluster(uint32_t local, int rank, float2 v) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(r), "f"(v.x), "f"(v.y) : "memory");
}

__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int NX, int NY, int KIND>
struct Resident {
  using Cfg = ResCfg<NX, NY, KIND>;
  using K = RegKind<KIND, 2>;
  static constexpr int C = Cfg::C, CG = K::CG, H = Cfg::H, HK = Cfg::HK, SP = Cfg::SP;

  const StepArgs& a;
  int b, rank, cl, rpc, rinv, nrow, rp, ka, kb, nc, pc, fs, nk, nr;  // nk / nr: kept / other columns this CTA has
  float2 *twx, *twy, *mid, *prod, *u, *q, *accA, *accB, *scr;
  float *kxs, *mrow, *kys, *ilap;
  float2* tabs;  // [4][lin_ch][nc][SP]: (c1, c5), (c6, c4), E2 - 1, E - 1; or (c1, c5) and c6 (floats)
  bool full;
  uint16_t* own;  // per column k < H: owner rank << 8 | local column

  __device__ __forceinline__ explicit Resident(const ResArgs& r) : a(r.a) {
    extern __shared__ float2 smem[];
    uint32_t v;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(v));
    rank = (int)v;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(v));
    cl = (int)v;
    b = (int)blockIdx.x / cl;
    ka = r.ka;
    kb = r.kb;
    pc = r.pc;
    fs = r.fs;
    nc = ka + kb;
    rpc = r.rpc;
    full = r.tables != 0;
    rinv = (65536 + rpc - 1) / rpc;  // x / rpc = x * rinv >> 16 for x < 256
    rp = rpc | 1;
    nk = min(ka, max(0, HK - rank * ka));
    nr = min(kb, max(0, H - HK - rank * kb));
    nrow = min(rpc, max(0, NX - rank * rpc));
    twx = smem;
    twy = twx + NX;
    mid = twy + NY;
    prod = mid + Cfg::NM * HK * rp;
    u = prod + Cfg::NP * NX * pc;
    q = u + C * nc * SP;
    accA = q + C * nc * SP;
    scr = accA + C * nc * SP;
    accB = u;
    if (fs > 1) {
      accB = scr;
      scr += C * nc * SP;
    }
    tabs = scr + (blockDim.x / 32) * Cfg::WS;
    ilap = (float*)tabs + (full ? 8 : 3) * a.lin_ch * nc * SP;
    kxs = ilap + (KIND == FSM_NL_LERAY ? nc * SP : 0);
    mrow = kxs + NX;
    kys = mrow + NX;
    own = (uint16_t*)(kys + 2 * ((H + 1) / 2));
  }

  // global column of local column i (i < nk: kept, nk <= i < nk + nr: the others)
  __device__ __forceinline__ int column(int i) const { return i < nk ? rank * ka + i : HK + rank * kb + (i - nk); }
  // the local slot (as the other CTAs address it) of local column i
  __device__ __forceinline__ int slot_of(int i) const { return i < nk ? i : ka + (i - nk); }

  __device__ __forceinline__ void load() {
    load_reg_twiddles<NX>(twx, a.tw, threadIdx.x, blockDim.x);
    load_reg_twiddles<NY>(twy, a.tw, threadIdx.x, blockDim.x);
    for (int x = threadIdx.x; x < NX; x += blockDim.x) {
      kxs[x] = a.kx[x];
      mrow[x] = (float)a.keepx[x] * a.scale;
    }
    for (int k = threadIdx.x; k < H; k += blockDim.x)
      own[k] = (uint16_t)(k < HK ? ((k / ka) << 8 | (k % ka)) : (((k - HK) / kb) << 8 | (ka + (k - HK) % kb)));
    for (int k = threadIdx.x; k < H; k += blockDim.x) kys[k] = a.ky[k];
    const int n = nk + nr, ts = a.lin_ch * nc * SP;
    for (int e = threadIdx.x; e < a.lin_ch * n * NX; e += blockDim.x) {
      const int i = e % n, x = (e / n) % NX, c = e / (n * NX);
      const float2* g = a.tab + (tab_batch(a, b) * a.lin_ch + c) * a.S + (int64_t)x * H + column(i);
      float2* d = tabs + (c * nc + slot_of(i)) * SP + x;
      // the SETDRK coefficients are real (k_phi_tables)
      d[0] = make_float2(g[2 * a.ts].x, g[4 * a.ts].x);
      if (full) {
        d[ts] = make_float2(g[5 * a.ts].x, g[3 * a.ts].x);
        d[2 * ts] = g[a.ts];
        d[3 * ts] = g[0];
      } else {
        ((float*)(tabs + ts))[(c * nc + slot_of(i)) * SP + x] = g[5 * a.ts].x;
      }
    }
    if (KIND == FSM_NL_LERAY) {
      for (int e = threadIdx.x; e < n * NX; e += blockDim.x) {
        const int i = e / NX, x = e % NX;
        ilap[slot_of(i) * SP + x] = inv_laplacian(a.kx[x], a.ky[column(i)], 0.f, 2);
      }
    }
    for (int e = threadIdx.x; e < C * n * NX; e += blockDim.x) {
      const int i = e % n, x = (e / n) % NX, c = e / (n * NX);
      u[(c * nc + slot_of(i)) * SP + x] = a.state[((int64_t)b * C + c) * a.S + (int64_t)x * H + column(i)];
    }
  }

  __device__ __forceinline__ void store() const {
    const int n = nk + nr;
    for (int e = threadIdx.x; e < C * n * NX; e += blockDim.x) {
      const int i = e % n, x = (e / n) % NX, c = e / (n * NX);
      a.state[((int64_t)b * C + c) * a.S + (int64_t)x * H + column(i)] = u[(c * nc + slot_of(i)) * SP + x];
    }
  }

  // The stage update of a column's points in the transform layout (registers v: N_s in, the next
  // stage's input out; STG -1, the priming pass: v = u): the recurrences of setdrk4_pre, with
  // exp(dt L / 2) u kept from stage 0 to stage 1 in u's place. Groups that share a column all read
  // the sums and one of them writes, so a stage then writes no array that it reads:
  //   stage   reads            writes                      (fs > 1)
  //     0     u                acc in A, q, e2u in B
  //     1     e2u in B, A      acc in u
  //     2     acc in u, q      acc in A
  //     3     acc in A         u
  // (fs == 1: B is u and acc stays in A.)
  template <int STG>
  __device__ __forceinline__ void update(float2 (&v)[Cfg::EX], int c, int slot, int col, int t, bool write, int frame) {
    constexpr int T = Cfg::TX, E = Cfg::EX;
    const int so = (c * nc + slot) * SP;
    float2* us = u + so;
    if (STG < 0) {
#pragma unroll
      for (int j = 0; j < E; ++j) v[j] = us[t + T * j];
    } else {
      float2 *qs = q + so, *as = accA + so, *e2s = accB + so;
      float2* a1s = fs > 1 ? us : as;  // acc between stages 1 and 2
      const int ts = a.lin_ch * nc * SP;
      const int to = ((a.lin_ch > 1 ? c : 0) * nc + slot) * SP;
      const float2* tab = tabs + to;
      const float* c6s = (const float*)(tabs + ts) + to;  // unless full
      const float2* tg = a.tab + (tab_batch(a, b) * a.lin_ch + (a.lin_ch > 1 ? c : 0)) * a.S + col;
      const float2* srcp = a.src ? a.src + ((int64_t)(a.src_batch > 1 ? b : 0) * C + c) * a.S + col : nullptr;
#pragma unroll
      for (int j = 0; j < E; ++j) {
        const int row = t + T * j;
        float2 nv = cscale(v[j], a.coef);
        if (srcp) nv = cadd(nv, srcp[(int64_t)row * H]);
        if (STG == 0) {
          const float2 c64 = full ? tab[ts + row] : make_float2(0.f, 0.f);
          const float2 Em1 = full ? tab[3 * ts + row] : tg[(int64_t)row * H];
          const float2 E2m1 = full ? tab[2 * ts + row] : tg[a.ts + (int64_t)row * H];
          const float2 c4 = full ? make_float2(c64.y, 0.f) : tg[3 * a.ts + (int64_t)row * H];
          const float2 c1 = make_float2(tab[row].x, 0.f);
          const float2 uu = us[row];
          const float2 e2u = cexpmul(E2m1, uu);
          const float2 a1 = cfma(c1, nv, e2u);
          const float2 acc = cfma(c4, nv, cexpmul(Em1, uu));
          const float2 qq = cfma(make_float2(-c1.x, -c1.y), nv, cexpmul(E2m1, a1));
          if (write) {
            as[row] = acc;
            qs[row] = qq;
            e2s[row] = e2u;
          }
          v[j] = a1;
        } else if (STG == 1 || STG == 2) {
          const float2 c15 = tab[row];
          const float2 c1 = make_float2(c15.x, 0.f), c5 = make_float2(c15.y, 0.f);
          const float2 acc = cfma(cscale(c5, 2.f), nv, STG == 1 ? as[row] : a1s[row]);
          v[j] = STG == 1 ? cfma(c1, nv, e2s[row]) : cfma(cscale(c1, 2.f), nv, qs[row]);
          if (write) (STG == 1 ? a1s : as)[row] = acc;
        } else {
          const float2 c6 = make_float2(full ? tab[ts + row].x : c6s[row], 0.f);
          v[j] = cfma(c6, nv, as[row]);
          if (write) us[row] = v[j];
        }
      }
    }
    if (write && frame >= 0) {
#pragma unroll
      for (int j = 0; j < E; ++j)
        a.traj[(((int64_t)b * a.n_frames + frame) * C + c) * a.S + (int64_t)(t + T * j) * H + col] = v[j];
    }
  }

  // stage: -1 primes; emit: build and send the next stage's fields; frame: record slot or -1
  __device__ __forceinline__ void columns(int stage, bool emit, int frame) {
    constexpr int T = Cfg::TX, E = Cfg::EX, GPW = 32 / T;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sub = lane / T, t = lane % T;
    const int groups = (blockDim.x >> 5) * GPW;
    const int n = nk + nr;
    const int per = (CG == 1 ? C : 1);  // items per column and sharing group
    const int items = n * per * fs;
    float2* sc = scr + warp * Cfg::WS + sub * reg_scratch<NX>();
#pragma unroll 1
    for (int base = warp * GPW; base < items; base += groups) {
      int item = base + sub;
      const bool act = item < items;
      item = act ? item : items - 1;
      // kept columns first: (share, channel, column) with the column fastest
      const int i = item % n, ch = (item / n) % per, share = item / (n * per);
      const int slot = slot_of(i), col = column(i);
      const bool write = act && share == 0;
      const bool send = emit && col < HK;
      float2 st[CG][E];
      if (stage >= 0) {
#pragma unroll
        for (int f = 0; f < CG; ++f) {
          const float2* src = prod + ((CG == 1 ? ch : f) * NX) * pc + slot;
#pragma unroll
          for (int j = 0; j < E; ++j) st[f][j] = src[(t + T * j) * pc];
          reg_fft<NX, false>(st[f], sc, twx, t);
        }
        if (KIND == FSM_NL_LERAY) {
#pragma unroll
          for (int j = 0; j < E; ++j) {
            const int row = t + T * j;
            PointK<2> pk;
            pk.kx = kxs[row];
            pk.ky = kys[col];
            pk.kz = 0.f;
            float2 nv[CG];
#pragma unroll
            for (int f = 0; f < CG; ++f) nv[f] = st[f][j];
            nv_leray_il<2, CG>(nv, pk, row, col, a, NX, ilap[slot * SP + row]);
#pragma unroll
            for (int f = 0; f < CG; ++f) st[f][j] = nv[f];
          }
        }
      }
#pragma unroll
      for (int f = 0; f < CG; ++f) {
        const int c = CG == 1 ? ch : f;
        switch (stage) {
          case 0: update<0>(st[f], c, slot, col, t, write, -1); break;
          case 1: update<1>(st[f], c, slot, col, t, write, -1); break;
          case 2: update<2>(st[f], c, slot, col, t, write, -1); break;
          case 3: update<3>(st[f], c, slot, col, t, write, frame); break;
          default: update<-1>(st[f], c, slot, col, t, write, frame); break;
        }
#pragma unroll
        for (int j = 0; j < E; ++j) st[f][j] = cscale(st[f][j], mrow[t + T * j]);
      }
      if (!__any_sync(0xffffffffu, send && act)) continue;
      const float ky = kys[col];
#pragma unroll
      for (int f = 0; f < CG; ++f) {
        const int c = CG == 1 ? ch : f;
        constexpr int NMC = (KIND == FSM_NL_VORTICITY) ? 4 : 2;  // fields of a channel
#pragma unroll 1
        for (int m = 0; m < NMC; m += fs) {  // fs divides NMC: the same count in every group of a warp
          const int mf = m + share;
          float2 v[E];
#pragma unroll
          for (int j = 0; j < E; ++j) {
            const float2 d = st[f][j];
            const float kxv = kxs[t + T * j];
            float2 x = d;
            if (KIND == FSM_NL_VORTICITY) {
              // 0: psi = -w/lap, 1: i kx psi, 2: w, 3: i kx w (selected without branches: the groups
              // of a warp may build different fields)
              const float lap = -(kxv * kxv + ky * ky);
              const float il = (lap == 0.f) ? 1.f : __fdividef(1.f, lap);
              x = cscale(d, mf < 2 ? -il : 1.f);
            }
            const float2 ix = cscale(cmuli(x), kxv);
            v[j] = (mf & 1) ? ix : x;
          }
          reg_fft<NX, true>(v, sc, twx, t);
          if (send && act) {
            const uint32_t m0 = smem_u32(mid + ((NMC * c + mf) * HK + col) * rp);
#pragma unroll
            for (int j = 0; j < E; ++j) {
              const int row = t + T * j;
              const int o = row * rinv >> 16;
              st_cluster(m0 + (uint32_t)(row - o * rpc) * 8u, o, v[j]);
            }
          }
        }
      }
    }
  }

  __device__ __forceinline__ void send_product(int f, int x, int k, float2 v) {
    const int o = own[k];
    st_cluster(smem_u32(prod + (f * NX + x) * pc + (o & 255)), o >> 8, v);
  }

  __device__ __forceinline__ void rows() {
    constexpr int T = Cfg::TY, E = Cfg::EY, GPW = 32 / T, J = NY / (2 * T);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sub = lane / T, t = lane % T;
    const int groups = (blockDim.x >> 5) * GPW;
    const int items = nrow;  // one row per group; vorticity pairs the rows of adjacent groups
    const int partner_lane = (lane & ~(T - 1)) | ((T - t) & (T - 1));
    float2* sc = scr + warp * Cfg::WS + sub * reg_scratch<NY>();
    const float2 zero = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int base = warp * GPW; base < items; base += groups) {
      int lr = base + sub;
      const bool act = lr < items;
      lr = act ? lr : (sub & 1);
      const int x = rank * rpc + lr;
      const float2* m0p = mid + lr;
      const int fstride = HK * rp;
      if (KIND == FSM_NL_VORTICITY) {
        float2 Z1[E], Z2[E];
#pragma unroll
        for (int j = 0; j < E; ++j) {
          Z1[j] = zero;
          Z2[j] = zero;
          if (reg_dead<NY, T, HK>(j)) continue;
          const int k = t + T * j;
          const bool hi = k > NY / 2;
          const int kk = hi ? NY - k : k;
          const bool selfc = (kk == 0) || (kk == NY / 2);
          const bool live = kk < HK;
          const float kyv = kys[kk];
          const int o = kk * rp;
          const float2 m0 = live ? m0p[o] : zero, m1 = live ? m0p[fstride + o] : zero;
          const float2 m2 = live ? m0p[2 * fstride + o] : zero, m3 = live ? m0p[3 * fstride + o] : zero;
          Z1[j] = herm_z(cscale(cmuli(m0), kyv), make_float2(-m1.x, -m1.y), selfc, hi);
          Z2[j] = herm_z(m3, cscale(cmuli(m2), kyv), selfc, hi);
        }
        reg_fft<NY, true>(Z1, sc, twy, t);
        reg_fft<NY, true>(Z2, sc, twy, t);
        // the product of this group's row and of its partner's (the other row of the pair)
#pragma unroll
        for (int j = 0; j < E; ++j) {
          const float p = Z1[j].x * Z2[j].x + Z1[j].y * Z2[j].y;
          const float o = __shfl_xor_sync(0xffffffffu, p, T);
          Z1[j] = (sub & 1) ? make_float2(o, p) : make_float2(p, o);
        }
        reg_fft<NY, false>(Z1, sc, twy, t);
#pragma unroll
        for (int j = 0; j <= J; ++j) {
          const float2 s = Z1[E - 1 - j];
          float2 recv;
          recv.x = __shfl_sync(0xffffffffu, s.x, partner_lane);
          recv.y = __shfl_sync(0xffffffffu, s.y, partner_lane);
          const float2 partner = (t == 0) ? Z1[(E - j) & (E - 1)] : recv;
          const int k = t + T * j;
          if (k <= NY / 2 && act) {
            const float2 zm = cconj(partner);
            const float2 val = (sub & 1) ? cscale(cmulmi(csub(Z1[j], zm)), 0.5f) : cscale(cadd(Z1[j], zm), 0.5f);
            send_product(0, x, k, val);
          }
        }
      } else {
        // convection, C = 2: conv_c = u0 dx u_c + u1 dy u_c
        float2 Z1[E], Z2[E];
#pragma unroll
        for (int j = 0; j < E; ++j) {
          Z1[j] = zero;
          Z2[j] = zero;
          if (reg_dead<NY, T, HK>(j)) continue;
          const int k = t + T * j;
          const bool hi = k > NY / 2;
          const int kk = hi ? NY - k : k;
          const bool selfc = (kk == 0) || (kk == NY / 2);
          const int o = kk * rp;
          if (kk < HK) {
            Z1[j] = herm_z(m0p[o], m0p[2 * fstride + o], selfc, hi);                 // u0 + i u1
            Z2[j] = herm_z(m0p[fstride + o], m0p[3 * fstride + o], selfc, hi);       // dx u0 + i dx u1
          }
        }
        reg_fft<NY, true>(Z1, sc, twy, t);
        reg_fft<NY, true>(Z2, sc, twy, t);
        float2 acc[E];
        float u1[E];
#pragma unroll
        for (int j = 0; j < E; ++j) {
          acc[j] = make_float2(Z1[j].x * Z2[j].x, Z1[j].x * Z2[j].y);
          u1[j] = Z1[j].y;
        }
#pragma unroll
        for (int j = 0; j < E; ++j) {
          Z2[j] = zero;
          if (reg_dead<NY, T, HK>(j)) continue;
          const int k = t + T * j;
          const bool hi = k > NY / 2;
          const int kk = hi ? NY - k : k;
          const bool selfc = (kk == 0) || (kk == NY / 2);
          const float kyv = kys[kk];
          const int o = kk * rp;
          if (kk < HK)
            Z2[j] = herm_z(cscale(cmuli(m0p[o]), kyv), cscale(cmuli(m0p[2 * fstride + o]), kyv), selfc, hi);
        }
        reg_fft<NY, true>(Z2, sc, twy, t);  // dy u0 + i dy u1
#pragma unroll
        for (int j = 0; j < E; ++j) {
          acc[j].x += u1[j] * Z2[j].x;
          acc[j].y += u1[j] * Z2[j].y;
        }
        reg_fft<NY, false>(acc, sc, twy, t);
#pragma unroll
        for (int j = 0; j <= J; ++j) {
          const float2 s = acc[E - 1 - j];
          float2 recv;
          recv.x = __shfl_sync(0xffffffffu, s.x, partner_lane);
          recv.y = __shfl_sync(0xffffffffu, s.y, partner_lane);
          const float2 partner = (t == 0) ? acc[(E - j) & (E - 1)] : recv;
          const int k = t + T * j;
          if (k <= NY / 2 && act) {
            const float2 zm = cconj(partner);
            send_product(0, x, k, cscale(cadd(acc[j], zm), 0.5f));
            send_product(1, x, k, cscale(cmulmi(csub(acc[j], zm)), 0.5f));
          }
        }
      }
    }
  }

  __device__ __forceinline__ void run() {
    load();
    cluster_sync();  // every CTA of the cluster runs before the first remote store
    columns(-1, a.steps > 0, a.slots ? a.slots[0] : -1);
#pragma unroll 1
    for (int step = 0; step < a.steps; ++step) {
      const int frame = a.slots ? a.slots[step + 1] : -1;
#pragma unroll 1
      for (int s = 0; s < 4; ++s) {
        cluster_sync();
        rows();
        cluster_sync();
        columns(s, !(s == 3 && step == a.steps - 1), s == 3 ? frame : -1);
      }
    }
    __syncthreads();
    store();
  }
};

template <int NX, int NY, int KIND>
__global__ void __launch_bounds__(kResThreads) k_plane_resident(const __grid_constant__ ResArgs r) {
  Resident<NX, NY, KIND> R(r);
  R.run();
}

// A kernel and what its launch needs, by grid size (fsm_resident_*.cu: one file per term).
struct ResKernel {
  void (*fn)(ResArgs);
  size_t (*smem)(int rpc, int ka, int kb, int pc, int fs, int tch, bool tables, int threads);
  int tx, ty;  // lanes per column / row group
};
ResKernel resident_vorticity(int nx, int ny);
ResKernel resident_convection(int nx, int ny);
ResKernel resident_leray(int nx, int ny);

template <int NX, int NY, int KIND>
ResKernel resident_entry() {
  using Cfg = ResCfg<NX, NY, KIND>;
  return {k_plane_resident<NX, NY, KIND>, Cfg::smem, Cfg::TX, Cfg::TY};
}

template <int NX, int KIND>
ResKernel resident_row(int ny) {
  switch (ny) {
    case 32: return resident_entry<NX, 32, KIND>();
    case 64: return resident_entry<NX, 64, KIND>();
    case 128: return resident_entry<NX, 128, KIND>();
    case 256: return resident_entry<NX, 256, KIND>();
  }
  return {};
}

template <int KIND>
ResKernel resident_kind(int nx, int ny) {
  switch (nx) {
    case 32: return resident_row<32, KIND>(ny);
    case 64: return resident_row<64, KIND>(ny);
    case 128: return resident_row<128, KIND>(ny);
    case 256: return resident_row<256, KIND>(ny);
  }
  return {};
}

}  // namespace fsm
