// The one-kernel leap-frog step of S right-hand sides, plane form: the step
// of k_rhs_step (mj_rhs_step.cuh), term for term and so with the same bits,
// where a thread owns an xy-plane k of an element for V right-hand sides.
//
// Phase 1 is bound by the shared-memory pipe, one 32-bit word per lane and
// cycle.  k_rhs_step's threads own z-lines and take every x- and y-neighbour
// of a point through shared memory: 4 n + 3 words per point and right-hand
// side.  A plane keeps u, vx and vy in registers (3 n^2 V of them); only u and
// vz cross planes, 2 n + 2 words (n + 5 with z-lines, below), and the factors
// and indices of a point, 8 words, serve V right-hand sides of a lane.  The
// largest V whose planes fit the 168 registers of 12 warps per SM (n = 7: 255
// of 7 to 8) was the fastest: V = 1 took 1.27 ms where V = 2 takes 1.07.
//
// The interior points of an element belong to no other one: phase 1 updates
// their dofs itself instead of writing and reading back their contributions,
// and the dof phase leaves them out (27 of 64 dofs at Q4, 125 of 216 at Q6).
//
// Step times, z-line form -> plane form (GB300): Q4 32^3, 64 sources 1313 ->
// 1067 us (element phase 862 -> 720, dof phase 442 -> 339); Q4 16^3, 16
// sources 53.1 -> 46.5; Q2 24^3, 64 sources 127.5 -> 91.0; Q3 24^3, 64 sources
// 269 -> 224; Q5 16^3, 64 sources 433 -> 342; Q6 14^3, 64 sources 487 -> 434,
// 8 sources on 10^3 30.4 -> 27.2.  What is left of phase 1 is the pipe at two
// thirds of its rate: 10 warps per SM wait for their gathers and for each
// other at the barriers.  (Tried and slower: gathers by cp.async during the
// previous tile's divergence, 1092; L2 prefetches of the next tile's rows,
// 1142.)
#pragma once
#include "mj_rhs_step.cuh"

namespace mj {

// ---- variants: (n, E, LB, V) per order -------------------------------------
// Only those that beat the z-line form's best: 8 right-hand sides stay with
// it at Q3 (28.4 us against 35.6 at 20^3) and Q5 (31.2 against 34.3 at 12^3),
// and whatever their number Q1 (its EN step takes 38 us against 31 at
// 27x23x20, 16 sources) and Q7, Q8 (3 n^2 registers).
#define MJ_RP_VARIANTS(X)                                                      \
  X(3, 16, 2, 4) X(3, 8, 4, 4) X(3, 4, 8, 4)                                   \
  X(4, 4, 8, 2) X(4, 2, 16, 2) X(4, 1, 32, 2)                                  \
  X(5, 4, 8, 1) X(5, 4, 8, 2) X(5, 2, 16, 2) X(5, 1, 32, 2)                    \
  X(6, 2, 16, 1) X(6, 1, 32, 1)                                                \
  X(7, 4, 8, 1) X(7, 2, 16, 1) X(7, 1, 32, 1)

namespace {

template <int N, int E, int LB, int V>
struct RpPlan {
  static constexpr int NN = N * N, Q = N * NN, Qp = elem_slots(N);
  static constexpr int T = E * N * LB;                              // threads
  static constexpr int W = LB * V;                                  // right-hand sides per pass
  static constexpr int I = N >= 4 ? N - 2 : 0, III = I * I * I;     // interior points (updated in phase 1)
  // Z-derivatives by z-lines, like the gather (a line of u is in a thread's registers there), instead of by planes from
  // shared memory: n + 5 words instead of 2 n + 2, one more barrier.  Q4: 16^3 x 16 49.7 -> 47.3 us, 32^3 x 64 with
  // LB = 8 1242 -> 1169, but 1069 -> 1110 with LB = 16.
  static constexpr bool kZLines = LB <= 8;
  static constexpr int Ip = (III + 3) / 4 * 4;
  static constexpr int kStageA = E * Qp * 32;                       // factors, Nodle and slots of a tile
  static constexpr int kStageB = kStageA + E * Ip * 4;              // and dt^2/D of its interior points
  static constexpr int kStage = (kStageB + 127) / 128 * 128;
  static constexpr int kWork = E * Q * W;                           // floats per work array
  static constexpr int kInner = E * III * W;                        // floats of 2 U^{n+1} - U^n at interior points
  static constexpr int kArea = (2 * kStage + 2 * kWork * 4 + kInner * 4 + 127) / 128 * 128;
  static constexpr int kSmem = kArea + 32;                          // + 4 mbarriers
  static constexpr int kHalf = kArea / 2 / 16 * 16;                 // one phase-2 chunk buffer
  static_assert(T % 32 == 0 && kWork % 4 == 0, "full warps, 16-byte arrays");
  // registers: three planes (u, vx, vy) of V values and about 45 more
  static constexpr int kRegs = (3 * NN * V + 45 + 7) / 8 * 8;
  static constexpr int kByRegs = 65536 / (T * (kRegs < 255 ? kRegs : 255));
  static constexpr int kBySmem = 228 * 1024 / (kSmem + 1024);
  static constexpr int kCtas = kByRegs < 1 ? 1 : kByRegs < kBySmem ? kByRegs : kBySmem < 1 ? 1 : kBySmem;
};

// The leap-frog update of one value, 2 u1 - u0 + md (-y) as the dof phase of
// k_rhs_step rounds it, in two parts.
__device__ __forceinline__ float rp_extrapolate(float u1, float u0) { return fmaf(2.f, u1, -u0); }
__device__ __forceinline__ float rp_update(float t, float md, float y) { return fmaf(md, -y, t); }

// c[a] of the derivative matrix, for the paired FMA (fma_v): one 8-byte
// constant holding the entry twice, where V is even.
__constant__ float2 c_gmat32x2[kMaxNK + 1][kMaxNK * kMaxNK];

template <int N, int V>
__device__ __forceinline__ void fma_g(float (&acc)[V], int idx, const float (&x)[V]) {
  if constexpr (V % 2 == 0) {
    const float2 c2 = c_gmat32x2[N][idx];
#pragma unroll
    for (int v = 0; v < V; v += 2) {
      const float2 r = __ffma2_rn(c2, make_float2(x[v], x[v + 1]), make_float2(acc[v], acc[v + 1]));
      acc[v] = r.x;
      acc[v + 1] = r.y;
    }
  } else {
    const float c = c_gmat32[N][idx];
#pragma unroll
    for (int v = 0; v < V; v++) acc[v] = fmaf(c, x[v], acc[v]);
  }
}

// Phase 2: sums, update and sources of this CTA's chunks, through two buffers
// of HALF bytes at smem and the two unused mbarriers at bar.
template <int T, int HALF, long SPIN>
__device__ __forceinline__ void rp_dof_phase(const RsParams& p, const RpParams& x, unsigned char* smem,
                                             uint64_t* bar, float* __restrict__ cur,
                                             const float* __restrict__ nxt, int par, int* err) {
  const int t = threadIdx.x, G = gridDim.x, S = p.S;
  float* dst = p.uout ? p.uout : cur;
  const int step = p.step >= 0 ? p.step : p.ctr[par];
  const bool pulse_on = step < p.n_pulse;
  const float pf = pulse_on ? (float)p.pulse[step] : 0.f;
  const int S4 = S >> 2;
  const unsigned magic = 0xffffffffu / (unsigned)S4 + 1u;  // item / S4 = umulhi(item, magic) below 2^16 items, S4 > 1
  auto issue_chunk = [&](int c, int b) {  // by warp 0, together
    if (c >= x.n_chunks) return;
    const RpChunk ch = x.chunks[c];
    const RpBuf L = rp_buf(ch.i0, ch.i1, ch.rows, S);
    unsigned char* base = smem + b * HALF;
    const int ia = ch.i0 & ~3;
    if (t == 0) {
      mbar_expect_tx(&bar[b], (uint32_t)L.end);
      bulk_g2s(base + L.m, x.mk + ia, (uint32_t)(L.p - L.m), &bar[b]);
      bulk_g2s(base + L.p, x.pk + ia, (uint32_t)(L.d - L.p), &bar[b]);
      bulk_g2s(base + L.d, x.dk + ia, (uint32_t)(L.end - L.d), &bar[b]);
    }
    __syncwarp();
    if (t < ch.s1 - ch.s0) {
      const RpSeg g = x.segs[ch.s0 + t];
      bulk_g2s(base + (size_t)g.ud * S * 4, nxt + (size_t)g.d0 * S, (uint32_t)(g.nd * S * 4), &bar[b]);
      bulk_g2s(base + L.u0 + (size_t)g.ud * S * 4, cur + (size_t)g.d0 * S, (uint32_t)(g.nd * S * 4), &bar[b]);
      bulk_g2s(base + L.r + (size_t)g.rd * S * 4, p.R + (size_t)g.q0 * S, (uint32_t)(g.nq * S * 4), &bar[b]);
    }
  };
  if (t < 32) {
    fence_proxy_async();         // phase-1 use of this shared memory is over
    fence_proxy_async_global();  // every CTA's R stores (ordered by the barrier) before the copies
    issue_chunk(blockIdx.x, 0);
    issue_chunk(blockIdx.x + G, 1);
  }
  // sources at interior dofs, one per (dof, right-hand side): phase 1 has stored their update without them
  if (pulse_on) {
    for (int e = blockIdx.x * T + t; e < x.n_fix; e += G * T) {
      const int d = __ldg(x.fix + 2 * e), r = __ldg(x.fix + 2 * e + 1);
      float un = dst[(size_t)d * S + r];
      un += __ldg(p.m + d) * pf * __ldg(x.fix_val + e);
      dst[(size_t)d * S + r] = un;
      if (p.ucopy) p.ucopy[(size_t)d * S + r] = un;
    }
  }
  uint32_t ph2 = 0u;
  for (int c = blockIdx.x, it = 0; c < x.n_chunks; c += G, ++it) {
    const int b = it & 1;
    const RpChunk ch = x.chunks[c];
    const bool ok = mbar_wait_bounded<SPIN>(&bar[b], (ph2 >> b) & 1u);
    if (__syncthreads_or(!ok)) {
      if (t == 0) {  // report; buffer b and, if issued, buffer b^1 may have copies in flight
        atomicExch(err, 1);
        mbar_wait_drain(&bar[b], (ph2 >> b) & 1u);
        if (c + G < x.n_chunks) mbar_wait_drain(&bar[b ^ 1], (ph2 >> (b ^ 1)) & 1u);
      }
      return;
    }
    ph2 ^= 1u << b;
    const unsigned char* buf = smem + b * HALF;
    const RpBuf L = rp_buf(ch.i0, ch.i1, ch.rows, S);
    const float4* su1 = reinterpret_cast<const float4*>(buf);
    const float4* su0 = reinterpret_cast<const float4*>(buf + L.u0);
    const float4* sR = reinterpret_cast<const float4*>(buf + L.r);
    const int sh = ch.i0 & 3;
    const float* sm = reinterpret_cast<const float*>(buf + L.m) + sh;
    const int* sp = reinterpret_cast<const int*>(buf + L.p) + sh;
    const int* sd = reinterpret_cast<const int*>(buf + L.d) + sh;
    const int q0 = sp[0];
    const int items = (ch.i1 - ch.i0) * S4;
    for (int item = t; item < items; item += 2 * T) {  // two items at a time: their loads overlap
      float4 y[2], o[2];
      int dl[2], c4[2], qa[2], nq[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int im = min(item + h * T, items - 1);
        dl[h] = (int)__umulhi((unsigned)im, magic);
        c4[h] = im - dl[h] * S4;
        qa[h] = sp[dl[h]];
        nq[h] = sp[dl[h] + 1] - qa[h];
        qa[h] = (qa[h] - q0) * S4 + c4[h];
        y[h] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      for (int i = 0; i < max(nq[0], nq[1]); i++)
#pragma unroll
        for (int h = 0; h < 2; h++)
          if (i < nq[h]) {
            const float4 r = sR[qa[h] + i * S4];
            y[h].x += r.x; y[h].y += r.y; y[h].z += r.z; y[h].w += r.w;
          }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const float4 a1 = su1[dl[h] * S4 + c4[h]], a0 = su0[dl[h] * S4 + c4[h]];
        const float md = sm[dl[h]];
        o[h] = make_float4(rp_update(rp_extrapolate(a1.x, a0.x), md, y[h].x),
                           rp_update(rp_extrapolate(a1.y, a0.y), md, y[h].y),
                           rp_update(rp_extrapolate(a1.z, a0.z), md, y[h].z),
                           rp_update(rp_extrapolate(a1.w, a0.w), md, y[h].w));
      }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        if (item + h * T >= items) break;
        const int d = sd[dl[h]];
        if (ch.has_src && pulse_on) {
          const float md = sm[dl[h]];
          float un[4] = {o[h].x, o[h].y, o[h].z, o[h].w};
          const int e1 = __ldg(p.src_ptr + d + 1);
          for (int e = __ldg(p.src_ptr + d); e < e1; e++) {
            const int r = __ldg(p.src_rhs + e);
            if ((r >> 2) == c4[h]) un[r & 3] += md * pf * __ldg(p.src_val + e);
          }
          o[h] = make_float4(un[0], un[1], un[2], un[3]);
        }
        *reinterpret_cast<float4*>(dst + (size_t)d * S + 4 * c4[h]) = o[h];
        if (p.ucopy) *reinterpret_cast<float4*>(p.ucopy + (size_t)d * S + 4 * c4[h]) = o[h];
      }
    }
    __syncthreads();  // buffer b is free
    if (t < 32) {
      fence_proxy_async();
      issue_chunk(c + 2 * G, b);
    }
  }
}

template <int N, int E, int LB, int V, bool EN, long SPIN = kSpinLimit>
__global__ void __launch_bounds__(RpPlan<N, E, LB, V>::T, RpPlan<N, E, LB, V>::kCtas)
    k_rhs_plane(const RsParams p, const RpParams x, SyncState* sync, int par, int* err,
                unsigned long long* __restrict__ stamps) {
  using P = RpPlan<N, E, LB, V>;
  constexpr int NN = P::NN, Q = P::Q, Qp = P::Qp, W = P::W, I = P::I;
  extern __shared__ __align__(128) unsigned char smem[];
  float* s_u = reinterpret_cast<float*>(smem + 2 * P::kStage);
  float* s_z = s_u + P::kWork;  // z-derivatives, then z-fluxes
  float* s_in = s_z + P::kWork;  // 2 U^{n+1} - U^n at the elements' interior points
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + P::kArea);
  float* s_ez = reinterpret_cast<float*>(smem + P::kSmem);  // EN: [el][source][z-line]
  const int t = threadIdx.x, G = gridDim.x, S = p.S;
  const int lb = t % LB;
  const int w = t / LB;
  const int el = w / N;
  const int k = w - el * N;                                // this thread's plane
  float* __restrict__ cur = par == 0 ? p.ua : p.ub;        // U^n, overwritten by U^{n+2}
  const float* __restrict__ nxt = par == 0 ? p.ub : p.ua;  // U^{n+1}
  float* dst = p.uout ? p.uout : cur;
  // step counters: ctr[1-par] = ctr[par] + 1 (phase 2 reads ctr[par] only)
  if (p.step < 0 && blockIdx.x == 0 && t == 0) p.ctr[1 - par] = p.ctr[par] + 1;
  // optional phase time stamps of this CTA: start, phase 1 done, barrier passed, end
  if (stamps && t == 0) stamps[4 * blockIdx.x] = global_ns();

  float gck[N], grk[N];
#pragma unroll
  for (int a = 0; a < N; a++) {
    gck[a] = c_gmat32[N][a * N + k];
    grk[a] = c_gmat32[N][k * N + a];
  }
  // work-array entry of point 0 of this thread's element and lane block; QS floats from a point to the next
  float* wu = s_u + (el * Q * LB + lb) * V;
  float* wz = s_z + (el * Q * LB + lb) * V;
  constexpr int QS = LB * V;
  float* wi = s_in + (el * P::III * LB + lb) * V;
  const int ki = k > 0 && k < N - 1 ? k - 1 : 0;  // its place among the planes with interior points
  const float* wi_k = wi + ki * I * I * QS;

  // ---- phase 1
  auto issue = [&](int st, int tile) {
    if (tile < p.n_tiles) {
      unsigned char* stage = smem + st * P::kStage;
      const bool in = I > 0 && x.interior;
      mbar_expect_tx(&bar[st], (uint32_t)(in ? P::kStageB : P::kStageA));
      bulk_g2s(stage, p.fac_e + (size_t)tile * E * 6 * Qp, (uint32_t)(E * Qp * 24), &bar[st]);
      bulk_g2s(stage + E * Qp * 24, p.nodle_e + (size_t)tile * E * Qp, (uint32_t)(E * Qp * 4), &bar[st]);
      bulk_g2s(stage + E * Qp * 28, p.slot_e + (size_t)tile * E * Qp, (uint32_t)(E * Qp * 4), &bar[st]);
      if (in) bulk_g2s(stage + P::kStageA, x.mi + (size_t)tile * E * P::Ip, (uint32_t)(E * P::Ip * 4), &bar[st]);
    }
  };
  if (t == 0) {
    for (int b = 0; b < 4; b++) mbar_init(&bar[b], 1);  // 0,1: tile stages; 2,3: chunk buffers
    fence_mbar_init();
    issue(0, blockIdx.x);
  }
  __syncthreads();
  uint32_t ph = 0u;
  for (int tile = blockIdx.x, it = 0; tile < p.n_tiles; tile += G, ++it) {
    const int s = it & 1;
    const bool ok = mbar_wait_bounded<SPIN>(&bar[s], (ph >> s) & 1u);
    if (__syncthreads_or(!ok)) {
      if (t == 0) {  // report; only stage s can have copies in flight here
        atomicExch(err, 1);
        mbar_wait_drain(&bar[s], (ph >> s) & 1u);
      }
      return;
    }
    ph ^= 1u << s;
    if (t == 0) {  // every thread is past the previous tile (barrier above): its stage is free
      fence_proxy_async();
      issue(s ^ 1, tile + G);
    }
    const float* f = reinterpret_cast<const float*>(smem + s * P::kStage) + el * 6 * Qp + k * NN;
    const int* nd0 = reinterpret_cast<const int*>(smem + s * P::kStage + E * Qp * 24);
    const int* nd = nd0 + el * Qp + k * NN;
    const int* st = nd + E * Qp;
    const float* mi = reinterpret_cast<const float*>(smem + s * P::kStage + P::kStageA) + el * P::Ip + ki * I * I;
    // interior points belong to no other element: their dofs are updated here (in the gather, k is the x index of
    // this thread's z-lines)
    const bool inner = x.interior && k > 0 && k < N - 1 && tile * E + el < x.n_elt;
    for (int pass = 0; pass < S / W; pass++) {
      const int col = pass * W + lb * V;
      if constexpr (P::kZLines) {
        // this thread's z-lines of its element: line (j = r, i = k) for every r
        float u[N][N][V], u0[I > 0 ? I : 1][I > 0 ? I : 1][V];
#pragma unroll
        for (int r = 0; r < N; r++)
#pragma unroll
          for (int a = 0; a < N; a++)
            vload_g<V>(nxt + (size_t)nd0[el * Qp + a * NN + r * N + k] * S + col, u[r][a]);
        if (I > 0 && inner) {
#pragma unroll
          for (int r = 0; r < I; r++)
#pragma unroll
            for (int a = 0; a < I; a++)
              vload<V>(cur + (size_t)nd0[el * Qp + (a + 1) * NN + (r + 1) * N + k] * S + col, u0[r][a]);
        }
        if (!EN && pass > 0) __syncthreads();  // the previous pass is done with s_z
#pragma unroll
        for (int r = 0; r < N; r++)
#pragma unroll
          for (int b = 0; b < N; b++) {
            float gz[V];
#pragma unroll
            for (int v = 0; v < V; v++) gz[v] = 0.f;
#pragma unroll
            for (int a = 0; a < N; a++) fma_g<N, V>(gz, a * N + b, u[r][a]);
            vstore<V>(wz + (b * NN + r * N + k) * QS, gz);
            vstore<V>(wu + (b * NN + r * N + k) * QS, u[r][b]);
          }
        if (I > 0 && inner) {
#pragma unroll
          for (int r = 0; r < I; r++)
#pragma unroll
            for (int a = 0; a < I; a++) {
#pragma unroll
              for (int v = 0; v < V; v++) u0[r][a][v] = rp_extrapolate(u[r + 1][a + 1][v], u0[r][a][v]);
              vstore<V>(wi + ((a * I + r) * I + k - 1) * QS, u0[r][a]);
            }
        }
      }
      float vx[NN][V], vy[NN][V];
      {
        float u[NN][V];
        if constexpr (P::kZLines) {
          __syncthreads();
#pragma unroll
          for (int q = 0; q < NN; q++) vload<V>(wu + (k * NN + q) * QS, u[q]);
        } else {
          float u0[I > 0 ? I * I : 1][V];
#pragma unroll
          for (int q = 0; q < NN; q++) vload_g<V>(nxt + (size_t)nd[q] * S + col, u[q]);
          if (I > 0 && inner) {
#pragma unroll
            for (int q = 0; q < I * I; q++) vload<V>(cur + (size_t)nd[(q / I + 1) * N + q % I + 1] * S + col, u0[q]);
          }
#pragma unroll
          for (int q = 0; q < NN; q++) vstore<V>(wu + (k * NN + q) * QS, u[q]);
          if (I > 0 && inner) {
#pragma unroll
            for (int q = 0; q < I * I; q++) {
#pragma unroll
              for (int v = 0; v < V; v++) u0[q][v] = rp_extrapolate(u[(q / I + 1) * N + q % I + 1][v], u0[q][v]);
              vstore<V>(wi + ((k - 1) * I * I + q) * QS, u0[q]);
            }
          }
          __syncthreads();
        }
        // the operation order of k_local_stiffness_rhs, written out as
        // explicit FMAs so all forms round alike
#pragma unroll
        for (int j = 0; j < N; j++)
#pragma unroll
          for (int i = 0; i < N; i++) {
            const int q = j * N + i;
            float gx[V], gy[V], gz[V];
#pragma unroll
            for (int v = 0; v < V; v++) gx[v] = gy[v] = gz[v] = 0.f;
            if constexpr (P::kZLines) vload<V>(wz + (k * NN + q) * QS, gz);
#pragma unroll
            for (int a = 0; a < N; a++) {
              if constexpr (!P::kZLines) {
                float rz[V];
                vload<V>(wu + (a * NN + q) * QS, rz);
                fma_v<V>(gz, gck[a], rz);
              }
              fma_g<N, V>(gx, a * N + i, u[j * N + a]);
              fma_g<N, V>(gy, a * N + j, u[a * N + i]);
            }
            const float bxx = f[q], bxy = f[Qp + q], bxz = f[2 * Qp + q];
            const float byy = f[3 * Qp + q], byz = f[4 * Qp + q], bzz = f[5 * Qp + q];
            float oz[V];
            mul_v<V>(vx[q], bxx, gx);
            fma_v<V>(vx[q], bxy, gy);
            fma_v<V>(vx[q], bxz, gz);
            mul_v<V>(vy[q], bxy, gx);
            fma_v<V>(vy[q], byy, gy);
            fma_v<V>(vy[q], byz, gz);
            mul_v<V>(oz, bxz, gx);
            fma_v<V>(oz, byz, gy);
            fma_v<V>(oz, bzz, gz);
            vstore<V>(wz + (k * NN + q) * QS, oz);  // over its own gz with z-lines
          }
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < N; j++)
#pragma unroll
        for (int i = 0; i < N; i++) {
          const int q = j * N + i;
          float y[V];
#pragma unroll
          for (int v = 0; v < V; v++) y[v] = 0.f;
#pragma unroll
          for (int a = 0; a < N; a++) {
            float rz[V];
            vload<V>(wz + (a * NN + q) * QS, rz);
            fma_g<N, V>(y, i * N + a, vx[j * N + a]);
            fma_g<N, V>(y, j * N + a, vy[a * N + i]);
            fma_v<V>(y, grk[a], rz);
          }
          float o[V];
#pragma unroll
          for (int v = 0; v < V; v++) o[v] = y[v];
          if (I > 0 && i > 0 && i < N - 1 && j > 0 && j < N - 1) {  // selects, no branches: they would part the loads
            const int qi = (j - 1) * I + i - 1;
            float un[V];
            vload<V>(wi_k + qi * QS, un);
            const float md = mi[qi];
#pragma unroll
            for (int v = 0; v < V; v++) o[v] = inner ? rp_update(un[v], md, 0.f + y[v]) : y[v];
            const size_t at = (size_t)(inner ? nd : st)[q] * S + col;
            vstore<V>((inner ? dst : p.R) + at, o);
            if (inner && p.ucopy) vstore<V>(p.ucopy + at, o);
          } else {
            vstore<V>(p.R + (size_t)st[q] * S + col, o);
          }
          if constexpr (EN) vstore<V>(wu + (k * NN + q) * QS, y);  // the gradients are done with u
        }
      if constexpr (EN) {  // z-lines of this tile: thread w takes lines w, w + E*N, ... of its sources
        float ue[N][N][V];  // loaded ahead of the barrier, for all lines
#pragma unroll
        for (int r = 0; r < N; r++) {
          const int ln = r * (E * N) + w, le = ln / NN, q = ln - le * NN;
#pragma unroll
          for (int a = 0; a < N; a++) vload_g<V>(p.ue + (size_t)nd0[le * Qp + a * NN + q] * S + col, ue[r][a]);
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < N; r++) {
          const int ln = r * (E * N) + w, le = ln / NN, q = ln - le * NN;
          float ez[V];
#pragma unroll
          for (int v = 0; v < V; v++) ez[v] = 0.f;
#pragma unroll
          for (int a = 0; a < N; a++) {
            float y[V];
            vload<V>(s_u + ((le * Q + a * NN + q) * LB + lb) * V, y);
#pragma unroll
            for (int v = 0; v < V; v++) ez[v] = fmaf(y[v], ue[r][a][v], ez[v]);
          }
#pragma unroll
          for (int v = 0; v < V; v++) s_ez[((size_t)le * S + col + v) * NN + q] = ez[v];
        }
        __syncthreads();  // s_u is free, s_ez complete
      }
    }
    if constexpr (EN) {  // one warp per element, in the order of k_rhs_step's EN form
      const int wq = t >> 5, l32 = t & 31;
      for (int e = wq; e < E; e += P::T / 32) {
        double acc = 0.0;
        for (int src = l32; src < S; src += 32) {
          const float* row = s_ez + ((size_t)e * S + src) * NN;
          float zs = 0.f;
          for (int q = 0; q < NN; q++) zs += row[q];
          acc += (double)zs;
        }
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
        if (l32 == 0) {
          const size_t ge = (size_t)tile * E + e;
          p.gacc[ge] += p.gcoef[ge] * acc;
        }
      }
    }
  }

  if constexpr (!EN) {
    if (p.rec_out) rs_receivers<P::T, P::kArea>(p, nxt, smem);
  }
  fence_proxy_async_global();  // this thread's R stores before the bulk copies of phase 2
  if (stamps && t == 0) stamps[4 * blockIdx.x + 1] = global_ns();
  if (!grid_barrier(sync, err)) return;
  if (stamps && t == 0) stamps[4 * blockIdx.x + 2] = global_ns();

  if constexpr (EN) asm volatile("griddepcontrol.launch_dependents;");  // the adjoint's injection may start
  // ---- phase 2
  rp_dof_phase<P::T, P::kHalf, SPIN>(p, x, smem, &bar[2], cur, nxt, par, err);
  if (stamps) {
    __syncthreads();
    if (t == 0) stamps[4 * blockIdx.x + 3] = global_ns();
  }
}

}  // namespace
}  // namespace mj
