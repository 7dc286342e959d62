// Many right-hand sides on one mesh (FP32): ONE cooperative persistent kernel
// per leap-frog step of all S runs.
//
//   phase 1  element tiles (E elements) of the mesh, persistent CTAs; the
//            factors and Nodle of a tile arrive by 1-D bulk copy (TMA) two
//            tiles ahead and stay in shared memory for all S/W passes.  A
//            thread owns a z-line of one element for V right-hand sides held
//            in registers (LB thread lanes x V = W right-hand sides per
//            pass), so every shared-memory line access moves V values at
//            once (8- or 16-byte loads) and the factors are read once per V.
//            The operation order per right-hand side is that of
//            k_local_stiffness_rhs; results go to the dof-ordered R.
//            (The plane form of the step, mj_rhs_plane.cuh, splits this phase
//            by planes instead.)
//   barrier  grid-wide, bounded (cooperative launch; mj_sync.cuh);
//   phase 2  dof chunks: u^{n+1}, u^n rows, the chunk's contiguous block of
//            R rows, dt^2/D and the CSR offsets arrive by bulk copy (two
//            buffers per CTA); then the sums, the leap-frog update and the
//            sources (grouped by dof) of every (dof, right-hand side).
// The variant (n, E, LB, V) is chosen at creation by timing the candidates
// of the order on the integrator itself.  The reference runs the S
// problems one after the other (MONTJOIE/src/Instationary/ModifiedEquation.cxx:290-345).
#include <cuda_runtime.h>

#include <algorithm>
#include <memory>
#include <vector>

#include "mj_rhs_step.cuh"

namespace mj {
namespace {

constexpr int kGraphStepsRs = 20;
constexpr int kRsSmallMesh = 6144;  // elements

// Order in which the threads of an element take its n*n z-lines.  A warp
// holds Z = 32/LB consecutive slots; each of its shared-memory line reads
// touches one x-line per distinct row j and one y-line per distinct column i
// among its z-lines.  Candidates: row-major, 2-D blocks, and strips of 2, 3 or
// 4 rows walked column by column, alternate strips in reverse (snake); the one
// with the fewest distinct rows + columns per warp, summed over the E
// elements of a tile, is kept (row-major on ties).  Every point's arithmetic
// is the same whichever thread does it.
void rs_zline_order(int n, int E, int LB, unsigned char* out) {
  const int Z = std::max(1, 32 / LB), NN = n * n;
  auto cost = [&](const std::vector<int>& ord) {
    int tot = 0;
    for (int w0 = 0; w0 < E * NN; w0 += Z) {
      std::vector<int> rows, cols;
      for (int sl = w0; sl < std::min(w0 + Z, E * NN); sl++) {
        const int e = sl / NN, q = ord[sl % NN];
        rows.push_back(e * n + q / n);
        cols.push_back(e * n + q % n);
      }
      std::sort(rows.begin(), rows.end());
      std::sort(cols.begin(), cols.end());
      tot += (int)(std::unique(rows.begin(), rows.end()) - rows.begin()) +
             (int)(std::unique(cols.begin(), cols.end()) - cols.begin());
    }
    return tot;
  };
  std::vector<std::vector<int>> cands;
  std::vector<int> ord;
  for (int q = 0; q < NN; q++) ord.push_back(q);
  cands.push_back(ord);
  {
    const int bw = Z >= 8 ? 4 : Z >= 2 ? 2 : 1, bh = std::max(1, Z / bw);
    ord.clear();
    for (int by = 0; by < n; by += bh)
      for (int bx = 0; bx < n; bx += bw)
        for (int y = by; y < std::min(by + bh, n); y++)
          for (int x = bx; x < std::min(bx + bw, n); x++) ord.push_back(y * n + x);
    cands.push_back(ord);
  }
  for (int bh = 2; bh <= 4; bh++) {
    ord.clear();
    for (int by = 0, strip = 0; by < n; by += bh, strip++)
      for (int c = 0; c < n; c++) {
        const int x = strip % 2 == 0 ? c : n - 1 - c;
        for (int y = by; y < std::min(by + bh, n); y++) ord.push_back(y * n + x);
      }
    cands.push_back(ord);
  }
  size_t best = 0;
  for (size_t c = 1; c < cands.size(); c++)
    if (cost(cands[c]) < cost(cands[best])) best = c;
  for (int q = 0; q < NN; q++) out[q] = (unsigned char)cands[best][q];
}



struct RsVariant {
  int n, E, LB, V, threads, smem, half;
  bool plane;  // the plane form (mj_rhs_plane.cuh)
};

const std::vector<RsVariant>& rs_variants() {
  static const std::vector<RsVariant> v = [] {
    std::vector<RsVariant> all = {
#define MJ_X(N_, E_, LB_, V_)                                                                                    \
  {N_, E_, LB_, V_, RsPlan<N_, E_, LB_, V_>::T, RsPlan<N_, E_, LB_, V_>::kSmem, RsPlan<N_, E_, LB_, V_>::kHalf, \
   false},
        MJ_RS_VARIANTS(MJ_X)
#undef MJ_X
    };
    for (const RpVariant& r : rp_variants()) all.push_back({r.n, r.E, r.LB, r.V, r.threads, 0, r.half, true});
    return all;
  }();
  return v;
}

int rs_prepare(const RsVariant& v, int S, int* ctas) {
  if (v.plane) return rp_prepare(v.n, v.E, v.LB, v.V, false, S, ctas);
#define MJ_X(N_, E_, LB_, V_)                                                                               \
  if (v.n == N_ && v.E == E_ && v.LB == LB_ && v.V == V_) {                                                 \
    MJ_CUDA(cudaFuncSetAttribute(k_rhs_step<N_, E_, LB_, V_>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                 v.smem));                                                                 \
    MJ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas, k_rhs_step<N_, E_, LB_, V_>, v.threads,    \
                                                          v.smem));                                        \
    return MJ_OK;                                                                                           \
  }
  MJ_RS_VARIANTS(MJ_X)
#undef MJ_X
  set_error("no many-source step variant");
  return MJ_ERR_ARG;
}

// A candidate's chunk lists (segs: the plane form's).
struct RsLists {
  DevBuf chunks, segs;
  int n_chunks = 0;
};

RpParams rp_params(const mj_lfb* b, const DevBuf& chunks, const DevBuf& segs, int n_chunks) {
  return {chunks.as<RpChunk>(),  segs.as<RpSeg>(),    b->rs_mi.as<float>(),
          b->rs_mk.as<float>(),  b->rs_pk.as<int>(),  b->rs_dk.as<int>(),
          b->rs_fix.as<int>(),   b->rs_fix_val.as<float>(), n_chunks,
          b->rs_n_fix,           b->op->n_elt,        b->rs_interior ? 1 : 0};
}

int rs_launch(const mj_lfb* b, const RsVariant& v, int grid, const RsParams& prm, const DevBuf& chunk_list,
              const DevBuf& segs, int n_chunks, int par, cudaStream_t s, unsigned long long* stamps = nullptr) {
  SyncState* sync = b->rs_sync.as<SyncState>();
  int* err = b->rs_err.as<int>();
  const RsChunk* chunks = chunk_list.as<RsChunk>();
  if (v.plane)
    return rp_launch(v.n, v.E, v.LB, v.V, false, grid, prm, rp_params(b, chunk_list, segs, n_chunks), sync, par, err,
                     s, stamps);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(v.threads);
  cfg.dynamicSmemBytes = v.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
#define MJ_X(N_, E_, LB_, V_)                                                                                \
  if (v.n == N_ && v.E == E_ && v.LB == LB_ && v.V == V_) {                                                  \
    MJ_CUDA(cudaLaunchKernelEx(&cfg, k_rhs_step<N_, E_, LB_, V_>, prm, chunks, n_chunks, sync, par, err,  \
                               stamps));                                                                     \
    count_launch();                                                                                          \
    return MJ_OK;                                                                                            \
  }
  MJ_RS_VARIANTS(MJ_X)
#undef MJ_X
  set_error("no many-source step variant");
  return MJ_ERR_ARG;
}

RsParams rs_params(mj_lfb* b, const RsVariant& v) {
  mj_op* op = b->op;
  RsParams p;
  p.fac_e = op->fac_e.as<float>();
  p.nodle_e = op->nodle_e.as<int>();
  p.slot_e = op->slot_e.as<int>();
  p.R = b->R.as<float>();
  p.ptr = op->ptr.as<int>();
  p.ua = b->ua.as<float>();
  p.ub = b->ub.as<float>();
  p.m = b->m.as<float>();
  p.pulse = b->pulse.as<double>();
  p.ctr = b->ctr.as<int>();
  p.src_ptr = b->rs_src_ptr.as<int>();
  p.src_rhs = b->rs_src_rhs.as<int>();
  p.src_val = b->rs_src_val.as<float>();
  p.uout = nullptr;
  p.ucopy = nullptr;
  p.ue = nullptr;
  p.gacc = nullptr;
  p.gcoef = nullptr;
  p.rec_idx = b->rec_idx.as<int>();
  p.rec_w = b->rec_w.as<double>();
  p.rec_out = nullptr;
  p.n_rec = b->n_rec;
  p.n_rec_w = b->n_rec_w;
  p.rec_stride = 0;
  p.n_pulse = b->n_pulse;
  p.S = b->S;
  p.n_tiles = op->n_elt_pad / v.E;
  p.step = -1;
  if (v.plane) return p;  // reads no z-line order
  if (b->rs_zmap_key[0] != v.n || b->rs_zmap_key[1] != v.E || b->rs_zmap_key[2] != v.LB) {
    rs_zline_order(v.n, v.E, v.LB, b->rs_zmap);
    b->rs_zmap_key[0] = v.n;
    b->rs_zmap_key[1] = v.E;
    b->rs_zmap_key[2] = v.LB;
  }
  std::copy(b->rs_zmap, b->rs_zmap + kMaxNK * kMaxNK, p.zmap);
  return p;
}

// Dof chunks of a variant: as many dofs as fit one phase-2 buffer (<= 512).
std::vector<RsChunk> rs_chunks(const mj_lfb* b, int half, const std::vector<char>& is_src) {
  const mj_op* op = b->op;
  const std::vector<int>& ptr = op->h_ptr;
  std::vector<RsChunk> out;
  for (int d = 0; d < op->n_dof;) {
    if (rs_buf(d, d + 1, ptr[d], ptr[d + 1], b->S).end > half) return {};
    int e = d + 1;
    while (e < op->n_dof && e - d < 512 && rs_buf(d, e + 1, ptr[d], ptr[e + 1], b->S).end <= half) e++;
    RsChunk ch = {d, e, ptr[d], ptr[e], 0, 0, 0, 0};
    for (int x = d; x < e; x++) ch.has_src |= is_src[x];
    out.push_back(ch);
    d = e;
  }
  return out;
}

// The dofs the plane form's dof phase updates (rs_h_dk, their first
// contribution rows rs_h_pk, device copies): all but the elements' interior
// ones, or all of them where an interior point shares its dof or the interior
// dofs are numbered in runs too short for the segments; and the sources at
// the dofs left out.  Order 3 and up: an order-2 element has one interior
// dof in eight of its own.
int rp_kept(mj_lfb* b, const std::vector<int>& dptr, const std::vector<int>& rhs, const std::vector<float>& val) {
  mj_op* op = b->op;
  const int n_dof = op->n_dof;
  std::vector<char> in(n_dof, 0);
  b->rs_interior = false;
  if (op->n >= 4) {
    DevBuf flag;
    MJ_CUDA(flag.alloc(sizeof(int) + n_dof));
    MJ_CUDA(cudaMemsetAsync(flag.ptr, 0, sizeof(int) + n_dof, b->stream));
    if (int rc = rp_mark_interior(op->nodle_e.as<int>(), op->ptr.as<int>(), op->n_elt, op->n,
                                  flag.as<char>() + sizeof(int), flag.as<int>(), b->stream))
      return rc;
    int bad = 0;
    MJ_CUDA(cudaMemcpyAsync(&bad, flag.ptr, sizeof(int), cudaMemcpyDeviceToHost, b->stream));
    MJ_CUDA(cudaMemcpyAsync(in.data(), flag.as<char>() + sizeof(int), n_dof, cudaMemcpyDeviceToHost, b->stream));
    MJ_CUDA(cudaStreamSynchronize(b->stream));
    long long kept = 0, runs = 0;
    for (int d = 0; d < n_dof; d++)
      if (!in[d]) {
        kept++;
        runs += d == 0 || in[d - 1];
      }
    b->rs_interior = !bad && kept >= 4 * runs;
    if (b->rs_interior) {
      const int I = op->n - 2;
      MJ_CUDA(b->rs_mi.alloc(sizeof(float) * (size_t)op->n_elt_pad * ((I * I * I + 3) / 4 * 4)));
      if (int rc = rp_interior_mass(op->nodle_e.as<int>(), b->m.as<float>(), op->n_elt, op->n_elt_pad, op->n,
                                    b->rs_mi.as<float>(), b->stream))
        return rc;
    } else {
      std::fill(in.begin(), in.end(), 0);
    }
  }
  std::vector<int>&dk = b->rs_h_dk, &pk = b->rs_h_pk;
  dk.clear();
  pk.assign(1, 0);
  std::vector<int> fix;
  std::vector<float> fix_val, mk, m(n_dof);
  MJ_CUDA(cudaMemcpy(m.data(), b->m.ptr, sizeof(float) * n_dof, cudaMemcpyDeviceToHost));
  for (int d = 0; d < n_dof; d++) {
    if (!in[d]) {
      dk.push_back(d);
      mk.push_back(m[d]);
      pk.push_back(pk.back() + op->h_ptr[d + 1] - op->h_ptr[d]);
      continue;
    }
    for (int e = dptr[d]; e < dptr[d + 1]; e++) {
      fix.push_back(d);
      fix.push_back(rhs[e]);
      fix_val.push_back(val[e]);
    }
  }
  b->rs_n_fix = (int)fix_val.size();
  auto upload = [](DevBuf& dst, const void* src, size_t bytes, size_t pad) {
    MJ_CUDA(dst.alloc(bytes + pad));
    MJ_CUDA(cudaMemset(dst.ptr, 0, bytes + pad));
    if (bytes) MJ_CUDA(cudaMemcpy(dst.ptr, src, bytes, cudaMemcpyHostToDevice));
    return MJ_OK;
  };
  if (int rc = upload(b->rs_mk, mk.data(), sizeof(float) * mk.size(), 32)) return rc;
  if (int rc = upload(b->rs_pk, pk.data(), sizeof(int) * pk.size(), 32)) return rc;
  if (int rc = upload(b->rs_dk, dk.data(), sizeof(int) * dk.size(), 32)) return rc;
  if (int rc = upload(b->rs_fix, fix.data(), sizeof(int) * fix.size(), 32)) return rc;
  return upload(b->rs_fix_val, fix_val.data(), sizeof(float) * fix_val.size(), 32);
}

// Chunks and segments of a plane variant: as many kept dofs as fit a buffer
// of half bytes (<= 512, <= kRpMaxSegs runs of consecutive dofs).
bool rp_chunks(const mj_lfb* b, int half, const std::vector<char>& is_src, std::vector<RpChunk>& out,
               std::vector<RpSeg>& segs) {
  const std::vector<int>&dk = b->rs_h_dk, &pk = b->rs_h_pk;
  const int n = (int)dk.size();
  for (int i0 = 0; i0 < n;) {
    if (rp_buf(i0, i0 + 1, pk[i0 + 1] - pk[i0], b->S).end > half) return false;
    RpChunk ch = {i0, i0, (int)segs.size(), 0, 0, 0, 0, 0};
    for (int i = i0; i < n && i - i0 < 512 && rp_buf(i0, i + 1, pk[i + 1] - pk[i0], b->S).end <= half; i++) {
      const int nq = pk[i + 1] - pk[i];
      if (i == i0 || dk[i] != dk[i - 1] + 1) {
        if ((int)segs.size() - ch.s0 == kRpMaxSegs) break;
        segs.push_back({dk[i], 0, b->op->h_ptr[dk[i]], 0, i - i0, pk[i] - pk[i0], 0, 0});
      }
      segs.back().nd++;
      segs.back().nq += nq;
      ch.i1 = i + 1;
      ch.has_src |= is_src[dk[i]];
    }
    ch.s1 = (int)segs.size();
    ch.rows = pk[ch.i1] - pk[i0];
    out.push_back(ch);
    i0 = ch.i1;
  }
  return true;
}

// The chunk lists of variant v on the device; L.n_chunks = 0 when a dof has
// too many contributions for one buffer.
int rs_lists(const mj_lfb* b, const RsVariant& v, const std::vector<char>& is_src, RsLists& L) {
  std::vector<RsChunk> ch;
  std::vector<RpChunk> pch;
  std::vector<RpSeg> segs;
  L.n_chunks = 0;
  if (v.plane ? !rp_chunks(b, v.half, is_src, pch, segs) : (ch = rs_chunks(b, v.half, is_src)).empty()) return MJ_OK;
  const void* src = v.plane ? (const void*)pch.data() : ch.data();
  const size_t bytes = v.plane ? sizeof(RpChunk) * pch.size() : sizeof(RsChunk) * ch.size();
  MJ_CUDA(L.chunks.alloc(bytes));
  MJ_CUDA(cudaMemcpy(L.chunks.ptr, src, bytes, cudaMemcpyHostToDevice));
  if (v.plane) {
    MJ_CUDA(L.segs.alloc(sizeof(RpSeg) * segs.size()));
    MJ_CUDA(cudaMemcpy(L.segs.ptr, segs.data(), sizeof(RpSeg) * segs.size(), cudaMemcpyHostToDevice));
  }
  L.n_chunks = (int)(v.plane ? pch.size() : ch.size());
  return MJ_OK;
}

void rs_use_lists(mj_lfb* b, RsLists& L) {
  std::swap(b->rs_chunks.ptr, L.chunks.ptr);
  std::swap(b->rs_chunks.bytes, L.chunks.bytes);
  std::swap(b->rs_segs.ptr, L.segs.ptr);
  std::swap(b->rs_segs.bytes, L.segs.bytes);
  b->rs_n_chunks = L.n_chunks;
}

// CTAs of a step: all that are resident, or as many as have work.  A small
// mesh's step is launch and grid barrier, and both grow with the CTAs: Q2
// 8x7x7 with 8 sources took 13 us on 608 CTAs and takes 8.5 on 60.
int rs_grid(int ctas, const RsParams& prm, int n_chunks) {
  return std::min(ctas * sm_count(), std::max(prm.n_tiles, n_chunks));
}

// The grid of a step that also takes the receivers' values.
int rs_rec_grid(const mj_lfb* b) {
  const int L = b->S % 32 == 0 ? 32 : b->S % 16 == 0 ? 16 : 8;
  return std::min(b->rs_resident, std::max(b->rs_grid, b->n_rec * (b->S / L)));
}

int rs_check_err(mj_lfb* b, cudaStream_t s) {
  int* herr = b->h_status.as<int>();
  MJ_CUDA(cudaMemcpyAsync(herr, b->rs_err.ptr, sizeof(int), cudaMemcpyDeviceToHost, s));
  MJ_CUDA(cudaStreamSynchronize(s));
  if (*herr) {
    cudaMemset(b->rs_err.ptr, 0, sizeof(int));
    cudaMemset(b->rs_sync.ptr, 0, sizeof(SyncState));
    set_error("mj_lfb_advance: a bounded wait of the step kernel timed out (state is invalid)");
    return MJ_ERR_STATE;
  }
  return MJ_OK;
}

}  // namespace

// Sources grouped by dof, chunk lists per candidate, and the variant choice:
// each candidate of the order runs 3 steps (after one warm-up) on the
// integrator's state, which mj_lfb_init resets afterwards.  The z-line
// variants are tried only where no plane variant runs (the plane form's list
// holds only variants faster than the best of them, mj_rhs_plane.cuh) and on
// meshes below kRsSmallMesh elements, where their smaller tiles use more of
// the SMs: 8.5 us against 9.5 at Q2 8x7x7 with 8 sources, 10.9 against 12.4
// at Q2 5x7x5 with 64, 32.2 against 34.4 at Q3 18^3 with 16; from 16^3 Q4 on
// the plane form's candidates are always ahead (45.0 against 49.9).  Leaves
// b->fused = false when no variant fits (S too large for a chunk buffer).
int lfb_fused_setup(mj_lfb* b) {
  mj_op* op = b->op;
  {
    // derivative matrix of this order into this unit's constant memory
    float v[kMaxNK * kMaxNK];
    for (int a = 0; a < op->n * op->n; a++) v[a] = (float)op->gradphi[a];
    MJ_CUDA(cudaMemcpyToSymbol(c_gmat32, v, sizeof(float) * op->n * op->n, sizeof(float) * kMaxNK * kMaxNK * op->n));
    if (int rc = rs_en_set_gmat(op->n, v)) return rc;
    if (int rc = rp_set_gmat(op->n, v)) return rc;
  }
  // sources grouped by dof: sorted (dof, rhs) pairs from the device copies
  std::vector<int> si(b->n_src), sr(b->n_src);
  std::vector<float> sv(b->n_src);
  if (b->n_src) {
    MJ_CUDA(cudaMemcpy(si.data(), b->src_idx.ptr, sizeof(int) * b->n_src, cudaMemcpyDeviceToHost));
    MJ_CUDA(cudaMemcpy(sr.data(), b->src_rhs.ptr, sizeof(int) * b->n_src, cudaMemcpyDeviceToHost));
    MJ_CUDA(cudaMemcpy(sv.data(), b->src_val.ptr, sizeof(float) * b->n_src, cudaMemcpyDeviceToHost));
  }
  std::vector<int> order(b->n_src);
  for (int t = 0; t < b->n_src; t++) order[t] = t;
  std::sort(order.begin(), order.end(), [&](int x, int y) { return si[x] != si[y] ? si[x] < si[y] : sr[x] < sr[y]; });
  std::vector<int> dptr((size_t)op->n_dof + 1, 0), rhs;
  std::vector<float> val;
  std::vector<char> is_src(op->n_dof, 0);
  for (int t = 0; t < b->n_src; t++) {
    const int e = order[t];
    rhs.push_back(sr[e]);
    val.push_back(sv[e]);
    is_src[si[e]] = 1;
    dptr[si[e] + 1]++;
  }
  for (int d = 0; d < op->n_dof; d++) dptr[d + 1] += dptr[d];
  MJ_CUDA(b->rs_src_ptr.alloc(sizeof(int) * dptr.size()));
  MJ_CUDA(b->rs_src_rhs.alloc(sizeof(int) * std::max<size_t>(1, rhs.size())));
  MJ_CUDA(b->rs_src_val.alloc(sizeof(float) * std::max<size_t>(1, val.size())));
  if (!rhs.empty()) {
    MJ_CUDA(cudaMemcpy(b->rs_src_rhs.ptr, rhs.data(), sizeof(int) * rhs.size(), cudaMemcpyHostToDevice));
    MJ_CUDA(cudaMemcpy(b->rs_src_val.ptr, val.data(), sizeof(float) * val.size(), cudaMemcpyHostToDevice));
  }
  MJ_CUDA(cudaMemcpy(b->rs_src_ptr.ptr, dptr.data(), sizeof(int) * dptr.size(), cudaMemcpyHostToDevice));
  MJ_CUDA(b->rs_sync.alloc(sizeof(SyncState)));
  MJ_CUDA(cudaMemset(b->rs_sync.ptr, 0, sizeof(SyncState)));
  MJ_CUDA(b->rs_err.alloc(sizeof(int)));
  MJ_CUDA(cudaMemset(b->rs_err.ptr, 0, sizeof(int)));

  int dev = 0, coop = 0;
  MJ_CUDA(cudaGetDevice(&dev));
  MJ_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
  b->fused = false;
  if (!coop) return MJ_OK;
  const std::vector<RsVariant>& all = rs_variants();
  cudaEvent_t e0, e1;
  MJ_CUDA(cudaEventCreate(&e0));
  MJ_CUDA(cudaEventCreate(&e1));
  const uint64_t before = launch_counter().load();
  double best = 1e300;
  int bi = -1;
  std::vector<RsLists> lists(all.size());
  std::vector<int> grids(all.size(), 0), resident(all.size(), 0);
  bool planes = false;  // a plane variant runs
  std::vector<size_t> tried(all.size());
  for (size_t c = 0; c < all.size(); c++) tried[c] = c;
  std::stable_partition(tried.begin(), tried.end(), [&](size_t c) { return all[c].plane; });
  for (size_t c : tried) {
    const RsVariant& v = all[c];
    if (!v.plane && planes && op->n_elt >= kRsSmallMesh) continue;
    if (v.n != op->n || b->S % (v.LB * v.V) != 0) continue;
    if (rs_buf(3, 4, 0, 8, b->S).end > v.half) continue;  // one dof (up to 8 contributions) must fit
    int ctas = 0;
    if (rs_prepare(v, b->S, &ctas) != MJ_OK || ctas < 1) continue;
    if (v.plane && b->rs_h_dk.empty())
      if (int rc = rp_kept(b, dptr, rhs, val)) return rc;
    if (int rc = rs_lists(b, v, is_src, lists[c])) return rc;
    if (!lists[c].n_chunks) continue;
    planes |= v.plane;
    const RsParams prm = rs_params(b, v);
    grids[c] = rs_grid(ctas, prm, lists[c].n_chunks);
    resident[c] = ctas * sm_count();
    auto run = [&](int k) {
      return rs_launch(b, v, grids[c], prm, lists[c].chunks, lists[c].segs, lists[c].n_chunks, k & 1, b->stream);
    };
    int rc = run(0);
    if (!rc) rc = cudaEventRecord(e0, b->stream) == cudaSuccess ? MJ_OK : MJ_ERR_CUDA;
    for (int k = 1; !rc && k <= 3; k++) rc = run(k);
    if (!rc) rc = cudaEventRecord(e1, b->stream) == cudaSuccess ? MJ_OK : MJ_ERR_CUDA;
    if (!rc) rc = rs_check_err(b, b->stream);
    float ms = 0.f;
    if (!rc) rc = cudaEventElapsedTime(&ms, e0, e1) == cudaSuccess ? MJ_OK : MJ_ERR_CUDA;
    if (rc) {
      cudaEventDestroy(e0);
      cudaEventDestroy(e1);
      return rc;
    }
    b->rs_tune_ms.push_back(ms / 3.0);
    b->rs_tune_variant.push_back((int)c);
    if (ms < best) {
      best = ms;
      bi = (int)c;
    }
  }
  launch_counter().store(before);  // tuning launches are not steps of the caller
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (bi < 0) return MJ_OK;
  b->rs_variant = bi;
  b->rs_threads = all[bi].threads;
  b->rs_grid = grids[bi];
  b->rs_resident = resident[bi];
  rs_use_lists(b, lists[bi]);
  b->fused = true;
  return MJ_OK;
}

// Forces the one-kernel step's variant (n of the operator, E, LB, V): its
// chunk list and persistent grid as the creation-time timing would set them;
// captured graphs of the previous variant are dropped.
int lfb_set_step_variant(mj_lfb* b, int E, int LB, int V) {
  mj_op* op = b->op;
  const std::vector<RsVariant>& all = rs_variants();
  int c = -1;
  for (size_t k = 0; k < all.size(); k++)
    if (all[k].n == op->n && all[k].E == E && all[k].LB == LB && all[k].V == V) c = (int)k;
  if (c < 0) {
    set_error("mj_lfb_set_step_variant: no one-kernel step variant with these parameters for this order");
    return MJ_ERR_ARG;
  }
  const RsVariant& v = all[c];
  if (b->S % (v.LB * v.V) != 0) {
    set_error("mj_lfb_set_step_variant: the number of right-hand sides is not a multiple of the variant's pass");
    return MJ_ERR_ARG;
  }
  int ctas = 0;
  if (int rc = rs_prepare(v, b->S, &ctas)) return rc;
  std::vector<char> is_src(op->n_dof, 0);
  if (b->n_src) {
    std::vector<int> si(b->n_src);
    MJ_CUDA(cudaMemcpy(si.data(), b->src_idx.ptr, sizeof(int) * b->n_src, cudaMemcpyDeviceToHost));
    for (int d : si) is_src[d] = 1;
  }
  RsLists lists;
  if (ctas >= 1 && !(v.plane && b->rs_h_dk.empty()))
    if (int rc = rs_lists(b, v, is_src, lists)) return rc;
  if (!lists.n_chunks) {
    set_error("mj_lfb_set_step_variant: the variant does not fit this integrator");
    return MJ_ERR_ARG;
  }
  rs_use_lists(b, lists);
  b->rs_variant = c;
  b->rs_threads = v.threads;
  b->rs_grid = rs_grid(ctas, rs_params(b, v), lists.n_chunks);
  b->rs_resident = ctas * sm_count();
  for (auto& g : b->rs_graph)
    if (g) {
      cudaGraphExecDestroy(g);
      g = nullptr;
    }
  b->fused = true;
  return MJ_OK;
}

// mj_lfb_advance with one cooperative kernel per step.  Without traces,
// runs of 20 steps replay a CUDA graph captured for the current step parity.
int lfb_fused_advance(mj_lfb* b, int nsteps, double* traces, int trace_stride, bool use_graph) {
  const RsVariant& v = rs_variants()[b->rs_variant];
  RsParams prm = rs_params(b, v);
  cudaStream_t s = b->stream;
  const bool diag = traces && b->n_rec;
  const bool prof = b->rs_profile;
  if (prof && b->rs_stamps.bytes < sizeof(unsigned long long) * 4 * b->rs_resident)
    MJ_CUDA(b->rs_stamps.alloc(sizeof(unsigned long long) * 4 * b->rs_resident));
  auto launch = [&](int par, cudaStream_t st) {
    return rs_launch(b, v, prm.rec_out ? rs_rec_grid(b) : b->rs_grid, prm, b->rs_chunks, b->rs_segs, b->rs_n_chunks,
                     par, st, prof ? b->rs_stamps.as<unsigned long long>() : (unsigned long long*)nullptr);
  };
  int done = 0;
  if (use_graph && !diag && !prof && nsteps >= kGraphStepsRs) {
    const int p0 = b->step & 1;
    if (!b->rs_graph[p0]) {
      cudaStream_t cs;
      MJ_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
      cudaGraph_t g;
      const uint64_t before = launch_counter().load();
      MJ_CUDA(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
      for (int k = 0; k < kGraphStepsRs; k++) {
        const int rc = launch((p0 + k) & 1, cs);
        if (rc) {
          cudaStreamEndCapture(cs, &g);
          cudaStreamDestroy(cs);
          return rc;
        }
      }
      MJ_CUDA(cudaStreamEndCapture(cs, &g));
      launch_counter().store(before);  // captured, not launched
      MJ_CUDA(cudaGraphInstantiate(&b->rs_graph[p0], g, 0));
      cudaGraphDestroy(g);
      cudaStreamDestroy(cs);
    }
    while (nsteps - done >= kGraphStepsRs) {
      MJ_CUDA(cudaGraphLaunch(b->rs_graph[p0], s));
      count_launch(kGraphStepsRs);
      done += kGraphStepsRs;
      b->step += kGraphStepsRs;
    }
  }
  for (; done < nsteps; done++) {
    // column `done` of the traces is the state before this step: the first by a kernel of its own, each other by the
    // step before it, which reads that state
    if (diag && done == 0) lfb_receivers(b, b->cur(), nsteps, 0, s);
    prm.rec_stride = nsteps;
    prm.rec_out = diag && done + 1 < nsteps ? b->traces_d.as<double>() + done + 1 : nullptr;
    const int rc = launch(b->step & 1, s);
    if (rc) return rc;
    b->cur_is_a = !b->cur_is_a;
    b->step++;
  }
  if (diag)
    if (int rc = lfb_copy_traces(b, nsteps, traces, trace_stride, s)) return rc;
  return rs_check_err(b, s);
}

// One step of the one-kernel form on caller-given states: U^n = u0,
// U^{n+1} = u1, U^{n+2} written to out (out may be u0); step: the pulse
// index, or -1 for a step without sources.  The integrator's own counter
// stays as it is.  Used by the adjoint's checkpoint replays and its adjoint
// steps.
int lfb_fused_step_on(mj_lfb* b, float* u0, float* u1, float* out, int step, cudaStream_t s) {
  const RsVariant& v = rs_variants()[b->rs_variant];
  RsParams prm = rs_params(b, v);
  prm.ua = u0;
  prm.ub = u1;
  prm.uout = out;
  prm.step = std::max(step, 0);
  if (step < 0) {
    prm.n_pulse = 0;
  }
  return rs_launch(b, v, b->rs_grid, prm, b->rs_chunks, b->rs_segs, b->rs_n_chunks, 0, s);
}

// lfb_fused_step_on without sources, in the EN form: also
// gacc[e] += gcoef[e] * sum_s sum_q ue[dof_q][s] (A_e u1)_q.  *done = false,
// with nothing launched, when the EN form of the step's variant does not fit
// (its shared memory grows with S); the caller then runs the plain step and
// the ENERGY kernel, which give the same bits.
int lfb_fused_step_en(mj_lfb* b, float* u0, float* u1, float* out, const float* ue, double* gacc,
                      const double* gcoef, cudaStream_t s, bool* done) {
  *done = false;
  const RsVariant& v = rs_variants()[b->rs_variant];
  if (b->rs_en_variant != b->rs_variant) {
    int ctas = 0;
    const int rc = v.plane ? rp_prepare(v.n, v.E, v.LB, v.V, true, b->S, &ctas)
                           : rs_en_prepare(v.n, v.E, v.LB, v.V, b->S, &ctas);
    if (rc) return rc;
    b->rs_en_variant = b->rs_variant;
    b->rs_en_grid = rs_grid(ctas, rs_params(b, v), b->rs_n_chunks);
  }
  if (b->rs_en_grid < 1) return MJ_OK;
  RsParams prm = rs_params(b, v);
  prm.ua = u0;
  prm.ub = u1;
  prm.uout = out;
  prm.n_pulse = 0;
  prm.step = 0;
  prm.ue = ue;
  prm.gacc = gacc;
  prm.gcoef = gcoef;
  SyncState* sync = b->rs_sync.as<SyncState>();
  int* err = b->rs_err.as<int>();
  const int rc = v.plane ? rp_launch(v.n, v.E, v.LB, v.V, true, b->rs_en_grid, prm,
                                     rp_params(b, b->rs_chunks, b->rs_segs, b->rs_n_chunks), sync, 0, err, s, nullptr)
                         : rs_en_launch(v.n, v.E, v.LB, v.V, b->S, b->rs_en_grid, prm, b->rs_chunks.as<RsChunk>(),
                                        b->rs_n_chunks, sync, 0, err, s);
  *done = rc == MJ_OK;
  return rc;
}

// Error flag of the one-kernel step (bounded waits), reset when set.
int lfb_fused_check(mj_lfb* b, cudaStream_t s) { return rs_check_err(b, s); }

// One ordinary step of the one-kernel form (the integrator's own states and
// step counter); copy: where a second copy of the new state goes, or nullptr;
// rec: where the receivers' values of U^{n+1} go (a column of an array of
// rec_stride columns).
int lfb_fused_step(mj_lfb* b, cudaStream_t s, float* copy, double* rec, int rec_stride) {
  const RsVariant& v = rs_variants()[b->rs_variant];
  RsParams prm = rs_params(b, v);
  prm.ucopy = copy;
  prm.rec_out = rec;
  prm.rec_stride = rec_stride;
  return rs_launch(b, v, rec ? rs_rec_grid(b) : b->rs_grid, prm, b->rs_chunks, b->rs_segs, b->rs_n_chunks, b->step & 1,
                   s);
}

// Phase times (ms) of the last profiled step: element phase (last CTA,
// mean CTA), barrier release, dof phase.
int lfb_phase_ms(const mj_lfb* b, double* out) {
  if (!b->rs_stamps.ptr) {
    set_error("mj_lfb_phase_ms: no profiled step has run (mj_lfb_profile)");
    return MJ_ERR_STATE;
  }
  const int grid = b->rs_grid;
  std::vector<unsigned long long> st(4 * (size_t)grid);
  MJ_CUDA(cudaMemcpy(st.data(), b->rs_stamps.ptr, sizeof(unsigned long long) * st.size(), cudaMemcpyDeviceToHost));
  unsigned long long t0 = ~0ull, p1max = 0, p2 = 0, end = 0;
  double p1sum = 0;
  for (int c = 0; c < grid; c++) t0 = std::min(t0, st[4 * c]);
  for (int c = 0; c < grid; c++) {
    p1max = std::max(p1max, st[4 * c + 1]);
    p1sum += double(st[4 * c + 1] - t0);
    p2 = std::max(p2, st[4 * c + 2]);
    end = std::max(end, st[4 * c + 3]);
  }
  out[0] = double(p1max - t0) * 1e-6;
  out[1] = p1sum / grid * 1e-6;
  out[2] = double(p2 - p1max) * 1e-6;
  out[3] = double(end - p2) * 1e-6;
  return MJ_OK;
}

}  // namespace mj
