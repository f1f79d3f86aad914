// Free-body Newton: the contact solve of pile worlds whose solver is Newton.
//
// Per env-step (newt_launch_pile_solo_step, pile_general.cu): pile_k_collide
// as for PGS (contacts, the active set, per contact the facet rows' J and M^-1 J^T and
// the row constants), then the solves here by the worlds' rows (a block of 32,
// 128 or 224 threads, or one warp past that), then pile_k_integrate
// with the velocity changes this kernel leaves (Euler, or RK4 with the
// solver's wrench held over the stages).
//
// The solve restates newt/src/solver.rs:1295-1407
// (solve_free_body_newton_impulses): the rows in contact order (four
// pyramidal facets per condim-3 contact), the dense response
// H_ij = J_i M^-1 J_j^T (column j of newt's matrix is every row's residual
// after a unit impulse on row j), the regulariser on its diagonal, the bias,
// and newt's NewtonSystem::solve with every row non-negative
// (newton_dense.cuh), then the bodies' velocity changes M^-1 J^T f (newt's
// wrenches J^T f / dt, integrated over dt).  H is formed from the records'
// J and M^-1 J^T triples: row i meets column j through every dynamic body
// the two contacts share.
//
// Scratch: past each world's pile scratch, H, its f32 factor, the FP64
// factor and the solver vectors, sized by the world's contact capacity
// (four rows per contact).
#include <algorithm>

#include "../../include/newt_gpu.h"
#include "newton_dense.cuh"
#include "pile_solver.cuh"
#include "quotient.cuh"

using namespace pile;

namespace {

// solver-record fields of pile_k_collide (pile_kernels.cu) that the solve reads
constexpr int S_BIAS = 40, S_REG = 52, S_MU = 53, S_ROWS = 60;

NEWT_HD int up4n(int n) { return (n + 3) / 4 * 4; }

// Newton region of one world, in floats past its pile scratch.
struct NewtonLay {
  int nrc;  // row capacity (4 x contact capacity, a multiple of 4)
  int H, LH, LHd, vec, order, words;
};
NEWT_HD NewtonLay newton_layout(int maxc) {
  NewtonLay n;
  n.nrc = up4n(4 * maxc);
  const int m = n.nrc * n.nrc;
  int f = 0;
  n.H = f; f += m;
  n.LH = f; f += m;
  n.LHd = f; f += 2 * m;    // doubles (the offset is a multiple of 16 floats)
  n.vec = f; f += 9 * n.nrc;  // x, b, d, g, p, s, u, v, breakpoints
  n.order = f; f += up4n(maxc);  // records in contact order (ints)
  n.words = (f + 31) / 32 * 32;
  return n;
}
NEWT_HD int pile_words(const WsLay& L) { return (L.nf + L.ni + 31) / 32 * 32; }

NEWT_D float dot4(float4 a, float4 b) { return (a.x * b.x + a.y * b.y) + a.z * b.z; }
NEWT_D float4 ldg4f(const float* p) { return *reinterpret_cast<const float4*>(p); }

// Rows the block kernel's instances hold (a thread per row), and the lists the
// first instance leaves the larger worlds in: one per instance after it, then
// the worlds of more rows than any holds.
constexpr int NB_SMALL = 32, NB_MID = 128, NB_BIG = 224;
struct NewtonLists { int* items; int* counts; int stride; };
NEWT_D int newton_class(int nr, int small) { return nr <= small ? -1 : nr <= NB_MID ? 0 : nr <= NB_BIG ? 1 : 2; }
// Active contacts of a world (islands are packed one after another).
NEWT_D int active_contacts(const WsLay& L, const int* wi) {
  const int nisl = wi[L.misc + 3];
  return nisl > 0 ? wi[L.istart + nisl - 1] + wi[L.icount + nisl - 1] : 0;
}

// A world of more than NB_BIG rows, one warp.
NEWT_D void newton_warp(const PileGroupDev& g, int w, int lane) {
  const WsLay L = ws_layout(g.nb, g.np, g.maxc);
  float* wf = g.scr + (size_t)w * g.sstride;
  int* wi = reinterpret_cast<int*>(wf + L.nf);
  const int nb = L.nb;
  const int nact = active_contacts(L, wi);
  const NewtonLay N = newton_layout(g.maxc);
  float* nw = wf + pile_words(L);
  const int ld = N.nrc, nr = 4 * nact;
  float* H = nw + N.H;
  float* LH = nw + N.LH;
  double* LHd = reinterpret_cast<double*>(nw + N.LHd);
  float* v = nw + N.vec;
  float *vx = v, *vb = v + ld, *vd = v + 2 * ld, *vg = v + 3 * ld, *vp = v + 4 * ld, *vs = v + 5 * ld,
        *vu = v + 6 * ld, *vv = v + 7 * ld, *vbrk = v + 8 * ld;
  int* ord = reinterpret_cast<int*>(nw + N.order);
  const int* sccon = wi + L.sccon;
  const float* sc0 = wf + L.sc;

  // records in contact order: record k's rank is the number of active
  // contacts with a smaller index (sccon holds them in island order)
  for (int k = lane; k < nact; k += 32) {
    const int c = sccon[k];
    int rank = 0;
    for (int q = 0; q < nact; ++q) rank += sccon[q] < c;
    ord[rank] = k;
  }
  __syncwarp();
  auto bodies = [&](int k, int* ba, int* bb) {
    const int* cc = wi + L.ci + CI * sccon[k];
    *ba = cc[2];
    *bb = cc[3];
  };
  // H (column-major, every entry: newt's matrix is J_i M^-1 J_j^T entry by
  // entry, its factor reads the lower triangle and its products the whole),
  // the bias and a zero-friction flag
  bool zero_mu = false;
  for (int e = lane; e < nr * nr; e += 32) {
    const int i = e % nr, j = e / nr;
    const int ki = ord[i >> 2], kj = ord[j >> 2];
    const float* ri = sc0 + (size_t)SC * ki + S_ROWS + 32 * (i & 3);       // J of row i
    const float* rj = sc0 + (size_t)SC * kj + S_ROWS + 32 * (j & 3) + 16;  // M^-1 J^T of row j
    int ia[2], ja[2];
    bodies(ki, &ia[0], &ia[1]);
    bodies(kj, &ja[0], &ja[1]);
    float h = 0.f;
    for (int si = 0; si < 2; ++si) {
      if (ia[si] >= nb) continue;  // a static side's row is zero
      for (int sj = 0; sj < 2; ++sj) {
        if (ja[sj] != ia[si]) continue;
        h += dot4(ldg4f(ri + 8 * si), ldg4f(rj + 8 * sj)) + dot4(ldg4f(ri + 8 * si + 4), ldg4f(rj + 8 * sj + 4));
      }
    }
    if (i == j) h += sc0[(size_t)SC * ki + S_REG];
    H[(size_t)j * ld + i] = h;
  }
  for (int i = lane; i < nr; i += 32) {
    const float* s = sc0 + (size_t)SC * ord[i >> 2];
    vb[i] = s[S_BIAS + (i & 3)];
    vx[i] = 0.f;
    zero_mu = zero_mu || s[S_MU] == 0.f;
  }
  zero_mu = __any_sync(dense::FULL, zero_mu);
  __syncwarp();
  const int iters = g.I[(size_t)w * g.lay.istride + g.lay.iters];
  uint32_t status = 0;
  dense::newton_solve(H, nr, ld, LH, ld, LHd, vx, vb, vd, vg, vp, vs, vu, vv, vbrk, iters, zero_mu, lane, &status);

  // the bodies' velocity changes M^-1 J^T f (world frame), and the impulses
  // to the contact records (the diagnostics surface)
  for (int b = lane; b < nb; b += 32) {
    float dvx = 0.f, dvy = 0.f, dvz = 0.f, dwx = 0.f, dwy = 0.f, dwz = 0.f;
    for (int i = 0; i < nr; ++i) {
      const int k = ord[i >> 2];
      int ba, bb;
      bodies(k, &ba, &bb);
      const float f = vx[i];
      const float* r = sc0 + (size_t)SC * k + S_ROWS + 32 * (i & 3) + 16;
      for (int s = 0; s < 2; ++s) {
        if ((s ? bb : ba) != b) continue;
        const float4 wl = ldg4f(r + 8 * s), wa = ldg4f(r + 8 * s + 4);
        dvx += wl.x * f; dvy += wl.y * f; dvz += wl.z * f;
        dwx += wa.x * f; dwy += wa.y * f; dwz += wa.z * f;
      }
    }
    st3(wf + L.dv + 3 * b, v3(dvx, dvy, dvz));
    st3(wf + L.dw + 3 * b, v3(dwx, dwy, dwz));
  }
  for (int i = lane; i < nr; i += 32) wf[L.con + CF * sccon[ord[i >> 2]] + C_IMP + (i & 3)] = vx[i];
  if (lane == 0 && status)
    atomicOr(reinterpret_cast<unsigned*>(g.I + (size_t)w * g.lay.istride + g.lay.status), status);
}

__global__ void __launch_bounds__(32) pile_k_newton_warp(const PileGroupDev* G, const int* wseg, int ng,
                                                         NewtonLists lists) {
  const int n = lists.counts[2];
  for (int k = blockIdx.x; k < n; k += gridDim.x) {
    const int t = lists.items[2 * lists.stride + k];
    const int gi = find_seg(wseg, ng, t);
    newton_warp(G[gi], t - wseg[gi], threadIdx.x);
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// Worlds of up to NB_BIG rows: a block per world, a thread per row
// ---------------------------------------------------------------------------
// What bounds it: one world's chain of dependent steps, its factor's columns
// and each direction's substitutions, with a few hundred worlds on the chip;
// one warp over matrices in global memory (pile_k_newton) spends them on L2
// and on scanning the rows a warp's width at a time.  Here
//   * H and its factor share one shared-memory matrix (H above, L below the
//     diagonal), rows of NB_LD floats so that float4 loads of eight rows meet
//     no bank twice;
//   * the factor advances four columns (a contact's rows) at a time, every
//     thread its row: four sums over the columns before, the 4 x 4 diagonal
//     factor by every thread for itself; the substitutions likewise;
//   * the line search sorts the breakpoints once.  Which coordinate leaves
//     when does not depend on the costs, so each leaving thread forms its own
//     H p and H s at that point from the ones before it, and a warp then
//     evaluates the windows side by side, their FP64 products a prefix sum
//     (an FP64 instruction occupies its pipe for sixteen cycles whether a
//     warp wants one value or 32).
// Three instances: 32 rows (a warp, twelve to an SM), 128 rows (whose shared
// matrix lets three blocks share an SM) and 224 (the most one SM holds).
// Measured (GB300, us an env-step, one warp per world -> by rows): 250 worlds
// of 10 boxes (24 to 108 rows) 1047 -> 130 (the solve 1000 -> 80), 500 of
// 16 boxes 2315 -> 340, 4000 of 5 boxes 761 -> 411, 20000 of 2 capsules
// 743 -> 510 (with 128 rows alone 1280: its blocks are three to an SM).

struct NbSmem { int cap, ld, m, di, v, x, p, s, brk, sx, sd, si, rec, ord, bod, red, flag, words; };
NEWT_HD NbSmem nb_smem(int rows) {
  NbSmem n;
  n.cap = rows;
  n.ld = 4 * ((n.cap / 4) | 1);
  int f = 0;
  n.red = f; f += rows / 32 * 8 * 2;  // doubles
  n.m = f; f += n.cap * n.ld;
  n.di = f; f += n.cap;
  n.v = f; f += n.cap;
  n.x = f; f += n.cap;
  n.p = f; f += n.cap;
  n.s = f; f += n.cap;
  n.brk = f; f += n.cap;
  n.sx = f; f += n.cap;
  n.sd = f; f += n.cap;
  n.si = f; f += n.cap;
  n.rec = f; f += 8 * n.cap;
  n.ord = f; f += n.cap / 4;
  n.bod = f; f += n.cap / 4;
  n.flag = f; f += 8;
  n.words = (f + 3) / 4 * 4;
  return n;
}

template <int ROWS>
NEWT_D void newton_block(const PileGroupDev& g, int w, float* nbs) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const WsLay L = ws_layout(g.nb, g.np, g.maxc);
  float* wf = g.scr + (size_t)w * g.sstride;
  int* wi = reinterpret_cast<int*>(wf + L.nf);
  const int nb = L.nb;
  const int nact = active_contacts(L, wi);
  const NewtonLay N = newton_layout(g.maxc);
  const NbSmem sm = nb_smem(ROWS);
  const int nr = 4 * nact, ld = sm.ld;
  float* M = nbs + sm.m;
  float *di = nbs + sm.di, *V = nbs + sm.v, *X = nbs + sm.x, *P = nbs + sm.p, *S = nbs + sm.s, *B = nbs + sm.brk,
        *SX = nbs + sm.sx, *SD = nbs + sm.sd, *R = nbs + sm.rec;
  int *SI = reinterpret_cast<int*>(nbs + sm.si), *ord = reinterpret_cast<int*>(nbs + sm.ord),
      *bod = reinterpret_cast<int*>(nbs + sm.bod);
  double* red = reinterpret_cast<double*>(nbs + sm.red);
  float* flag = nbs + sm.flag;
  const int* sccon = wi + L.sccon;
  const float* sc0 = wf + L.sc;
  auto f4 = [](const float* q) { return *reinterpret_cast<const float4*>(q); };

  // records in contact order, and their bodies (nb: a static side)
  for (int k = tid; k < nact; k += ROWS) {
    const int c = sccon[k];
    int rank = 0;
    for (int q = 0; q < nact; ++q) rank += sccon[q] < c;
    const int* cc = wi + L.ci + CI * c;
    ord[rank] = k;
    bod[rank] = cc[2] | cc[3] << 16;
  }
  __syncthreads();
  // H's lower triangle, a thread per pair of contacts, stored above the
  // diagonal: entry (i, j) = J_i M^-1 J_j^T, i >= j, at M[j][i]
  for (int a = 0, b = tid;; b += ROWS) {
    while (a < nact && b > a) b -= ++a;
    if (a >= nact) break;
    const int wa = bod[a], wb = bod[b];
    const int ia[2] = {wa & 0xffff, wa >> 16}, jb[2] = {wb & 0xffff, wb >> 16};
    float h[4][4] = {};
    const float* ra = sc0 + (size_t)SC * ord[a] + S_ROWS;
    const float* rb = sc0 + (size_t)SC * ord[b] + S_ROWS + 16;
    for (int si = 0; si < 2; ++si) {
      if (ia[si] >= nb) continue;  // a static side's row is zero
      for (int sj = 0; sj < 2; ++sj) {
        if (jb[sj] != ia[si]) continue;
        float4 jl[4], ja[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          jl[i] = ldg4f(ra + 32 * i + 8 * si);
          ja[i] = ldg4f(ra + 32 * i + 8 * si + 4);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 ml = ldg4f(rb + 32 * j + 8 * sj), ma = ldg4f(rb + 32 * j + 8 * sj + 4);
#pragma unroll
          for (int i = 0; i < 4; ++i) h[i][j] += dot4(jl[i], ml) + dot4(ja[i], ma);
        }
      }
    }
    const float reg = a == b ? sc0[(size_t)SC * ord[a] + S_REG] : 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (a != b || i >= j) M[(4 * b + j) * ld + 4 * a + i] = h[i][j] + (a == b && i == j ? reg : 0.f);
  }
  const int r = tid;
  const bool in = r < nr;
  float bias = 0.f;
  bool zero_mu = false;
  if (in) {
    const float* s = sc0 + (size_t)SC * ord[r >> 2];
    bias = s[S_BIAS + (r & 3)];
    zero_mu = s[S_MU] == 0.f;
  }
  __syncthreads();
  const float hd = in ? M[r * ld + r] : 1.f;
  float* row = M + (in ? r : nr - 1) * ld;

  // ---- L L^T = H, four columns at a time ----
  float mn = 1e30f, mx = 0.f;
  bool ok = true;
  for (int p = 0; p < nr; p += 4) {
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    if (in && r >= p) {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (r >= p + u) s[u] = M[(p + u) * ld + r];
      for (int k = 0; k < p; k += 4) {
        const float4 a = f4(row + k);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float4 c = f4(M + (p + u) * ld + k);
          s[u] = fmaf(-a.x, c.x, s[u]);
          s[u] = fmaf(-a.y, c.y, s[u]);
          s[u] = fmaf(-a.z, c.z, s[u]);
          s[u] = fmaf(-a.w, c.w, s[u]);
        }
      }
      if (r < p + 4) *reinterpret_cast<float4*>(R + 4 * (r - p)) = make_float4(s[0], s[1], s[2], s[3]);
    }
    __syncthreads();
    const float4 d0 = f4(R), d1 = f4(R + 4), d2 = f4(R + 8), d3 = f4(R + 12);
    const float l00 = sqrtf(d0.x), i0 = 1.f / l00;
    const float l10 = d1.x * i0, l20 = d2.x * i0, l30 = d3.x * i0;
    const float e11 = fmaf(-l10, l10, d1.y), l11 = sqrtf(e11), i1 = 1.f / l11;
    const float l21 = fmaf(-l20, l10, d2.y) * i1, l31 = fmaf(-l30, l10, d3.y) * i1;
    const float e22 = fmaf(-l21, l21, fmaf(-l20, l20, d2.z)), l22 = sqrtf(e22), i2 = 1.f / l22;
    const float l32 = fmaf(-l31, l21, fmaf(-l30, l20, d3.z)) * i2;
    const float e33 = fmaf(-l32, l32, fmaf(-l31, l31, fmaf(-l30, l30, d3.w))), l33 = sqrtf(e33), i3 = 1.f / l33;
    ok = ok && d0.x > 0.f && e11 > 0.f && e22 > 0.f && e33 > 0.f;
    mn = fminf(fminf(mn, fminf(l00, l11)), fminf(l22, l33));
    mx = fmaxf(fmaxf(mx, fmaxf(l00, l11)), fmaxf(l22, l33));
    if (in && r >= p + 4) {
      const float y0 = s[0] * i0, y1 = fmaf(-y0, l10, s[1]) * i1;
      const float y2 = fmaf(-y1, l21, fmaf(-y0, l20, s[2])) * i2;
      const float y3 = fmaf(-y2, l32, fmaf(-y1, l31, fmaf(-y0, l30, s[3]))) * i3;
      *reinterpret_cast<float4*>(row + p) = make_float4(y0, y1, y2, y3);
    } else if (r >= p && in) {
      const int q = r - p;
      row[p] = q == 0 ? l00 : q == 1 ? l10 : q == 2 ? l20 : l30;
      if (q > 0) row[p + 1] = q == 1 ? l11 : q == 2 ? l21 : l31;
      if (q > 1) row[p + 2] = q == 2 ? l22 : l32;
      if (q > 2) row[p + 3] = l33;
      di[r] = q == 0 ? i0 : q == 1 ? i1 : q == 2 ? i2 : i3;
    }
    __syncthreads();
  }

  // H times the shared vectors a and b, this thread's row: H above the
  // diagonal lies in its column up to the warp's rows, in its row past them
  auto products = [&](const float* a, const float* b, float* oa, float* ob) {
    float sa = 0.f, sb = 0.f;
    const int lo = 32 * warp, hi = min(lo + 32, nr);
    const float* col = M + r;
#pragma unroll 4
    for (int c = 0; c < lo; ++c) {
      const float h = col[c * ld];
      sa = fmaf(h, a[c], sa);
      sb = fmaf(h, b[c], sb);
    }
#pragma unroll 4
    for (int c = lo; c < hi; ++c) {
      const float h = c == r ? hd : c < r ? col[c * ld] : row[c];
      sa = fmaf(h, a[c], sa);
      sb = fmaf(h, b[c], sb);
    }
    for (int c = hi; c < nr; c += 4) {
      const float4 h = f4(row + c), va = f4(a + c), vb = f4(b + c);
      sa = fmaf(h.x, va.x, sa); sb = fmaf(h.x, vb.x, sb);
      sa = fmaf(h.y, va.y, sa); sb = fmaf(h.y, vb.y, sb);
      sa = fmaf(h.z, va.z, sa); sb = fmaf(h.z, vb.z, sb);
      sa = fmaf(h.w, va.w, sa); sb = fmaf(h.w, vb.w, sb);
    }
    *oa = sa;
    *ob = sb;
  };

  const int iters = g.I[(size_t)w * g.lay.istride + g.lay.iters];
  uint32_t status = 0;
  float x = 0.f;
  if (!ok || (mx / mn) * (mx / mn) > 1.0e6f) {
    // the FP64 factor (or newt's zero-friction pivot): the general solve, one warp
    float* nw = wf + pile_words(L);
    const int nrc = N.nrc;
    float* H = nw + N.H;
    float* v = nw + N.vec;
    zero_mu = __syncthreads_or(zero_mu);
    if (in) {
      for (int c = 0; c < nr; ++c) H[(size_t)c * nrc + r] = c == r ? hd : c < r ? M[c * ld + r] : row[c];
      v[r] = 0.f;
      v[nrc + r] = bias;
    }
    __syncthreads();
    if (warp == 0)
      dense::newton_solve(H, nr, nrc, nw + N.LH, nrc, reinterpret_cast<double*>(nw + N.LHd), v, v + nrc, v + 2 * nrc,
                          v + 3 * nrc, v + 4 * nrc, v + 5 * nrc, v + 6 * nrc, v + 7 * nrc, v + 8 * nrc, iters,
                          zero_mu, lane, &status);
    __syncthreads();
    if (in) x = v[r];
  } else {
    const int max_it = iters > 1 ? iters : 1;
    int done = 0;
    double cur = 0.0;
    for (int it = 0; it < max_it; ++it) {
      float hx = 0.f, dummy;
      if (it > 0) {
        if (in) X[r] = x;
        __syncthreads();
        if (in) products(X, X, &hx, &dummy);
      }
      const float grad = in ? hx + bias : 0.f;
      // d = -(L L^T)^-1 grad
      float d = -grad;
      if (in) V[r] = d;
      __syncthreads();
      for (int p = 0; p < nr; p += 4) {
        const float4 v = f4(V + p), i = f4(di + p);
        const float l00 = M[p * ld + p];
        const float4 l1 = f4(M + (p + 1) * ld + p), l2 = f4(M + (p + 2) * ld + p), l3 = f4(M + (p + 3) * ld + p);
        const float y0 = quot(v.x, l00, i.x);
        const float y1 = quot(fmaf(-l1.x, y0, v.y), l1.y, i.y);
        const float y2 = quot(fmaf(-l2.y, y1, fmaf(-l2.x, y0, v.z)), l2.z, i.z);
        const float y3 = quot(fmaf(-l3.z, y2, fmaf(-l3.y, y1, fmaf(-l3.x, y0, v.w))), l3.w, i.w);
        if (in && r >= p + 4) {
          const float4 l = f4(row + p);
          d = fmaf(-l.x, y0, d);
          d = fmaf(-l.y, y1, d);
          d = fmaf(-l.z, y2, d);
          d = fmaf(-l.w, y3, d);
          if (r < p + 8) V[r] = d;
        } else if (r >= p) {
          d = r == p ? y0 : r == p + 1 ? y1 : r == p + 2 ? y2 : y3;
        }
        __syncthreads();
      }
      if (in && r >= nr - 4) V[r] = d;
      __syncthreads();
      for (int p = nr - 4; p >= 0; p -= 4) {
        const float4 v = f4(V + p), i = f4(di + p);
        const float l00 = M[p * ld + p];
        const float4 l1 = f4(M + (p + 1) * ld + p), l2 = f4(M + (p + 2) * ld + p), l3 = f4(M + (p + 3) * ld + p);
        const float z3 = quot(v.w, l3.w, i.w);
        const float z2 = quot(fmaf(-l3.z, z3, v.z), l2.z, i.z);
        const float z1 = quot(fmaf(-l2.y, z2, fmaf(-l3.y, z3, v.y)), l1.y, i.y);
        const float z0 = quot(fmaf(-l1.x, z1, fmaf(-l2.x, z2, fmaf(-l3.x, z3, v.x))), l00, i.x);
        if (r < p) {
          const float* c = M + p * ld + r;
          d = fmaf(-c[3 * ld], z3, d);
          d = fmaf(-c[2 * ld], z2, d);
          d = fmaf(-c[ld], z1, d);
          d = fmaf(-c[0], z0, d);
          if (r >= p - 4) V[r] = d;
        } else if (r < p + 4) {
          d = r == p ? z0 : r == p + 1 ? z1 : r == p + 2 ? z2 : z3;
        }
        __syncthreads();
      }
      if (!in) d = 0.f;
      // ---- exact line search over the projected path (newton.rs:435-556) ----
      const bool fr = x > 0.f || (x == 0.f && d > 0.f);
      const float p0 = fr ? x : 0.f, s0 = fr ? d : 0.f;
      const float a0 = (x > 0.f && d < 0.f) ? -x / d : 2.f;
      const float brk = (a0 > 0.f && a0 < 1.f) ? a0 : 2.f;
      const float gd = dense::warp_sum(grad * d);
      if (lane == 0) flag[warp] = gd;
      if (in) {
        P[r] = p0;
        S[r] = s0;
        B[r] = brk;
      }
      const int nbrk = __syncthreads_count(brk < 1.f);
      float slope = 0.f;
      for (int q = 0; q < ROWS / 32; ++q) slope += flag[q];
      if (slope >= 0.f) break;
      float u = 0.f, v = 0.f;
      if (in) {
        if (it > 0) products(P, S, &u, &v);
        else products(S, S, &v, &dummy);  // x = 0: p = 0
      }
      {
        double s8[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        if (32 * warp < nr) {
          if (it > 0) {
            s8[0] = (double)p0 * (double)u;
            s8[1] = (double)p0 * (double)v;
            s8[3] = (double)bias * (double)p0;
            s8[5] = (double)x * (double)hx;
            s8[6] = (double)x * (double)bias;
          }
          s8[2] = (double)s0 * (double)v;
          s8[4] = (double)bias * (double)s0;
          dense::warp_sums(s8, lane);
        }
        if (lane == 0)
          for (int q = 0; q < 8; ++q) red[8 * warp + q] = s8[q];
      }
      // the breakpoints in order (ties: the smaller row first)
      int rank = -1;
      if (brk < 1.f) {
        rank = 0;
        for (int c = 0; c < nr; c += 4) {
          const float4 o = f4(B + c);
          rank += (o.x < brk || (o.x == brk && c < r)) + (o.y < brk || (o.y == brk && c + 1 < r)) +
                  (o.z < brk || (o.z == brk && c + 2 < r)) + (o.w < brk || (o.w == brk && c + 3 < r));
        }
        SX[rank] = p0;
        SD[rank] = s0;
        SI[rank] = r;
      }
      __syncthreads();
      if (rank >= 0) {
        float uj = u, vj = v;  // H p and H s at this row once the earlier ones have left
        for (int m = 0; m < rank; ++m) {
          const int c = SI[m];
          const float h = M[min(c, r) * ld + max(c, r)];
          uj = fmaf(-SX[m], h, uj);
          vj = fmaf(-SD[m], h, vj);
        }
        float* o = R + 8 * rank;
        o[0] = brk; o[1] = p0; o[2] = s0; o[3] = uj; o[4] = vj; o[5] = bias; o[6] = hd;
      }
      __syncthreads();
      if (warp == 0) {
        double c5[5];  // p.Hp, p.Hs, s.Hs, b.p, b.s
        double xhx = 0.0, xb = 0.0;
        for (int q = 0; q < 5; ++q) c5[q] = 0.0;
        for (int q = 0; 32 * q < nr; ++q) {
          for (int k = 0; k < 5; ++k) c5[k] += red[8 * q + k];
          xhx += red[8 * q + 5];
          xb += red[8 * q + 6];
        }
        cur = 0.5 * xhx + xb;
        float best_a = 0.f;
        double best_c = cur;
        for (int base = 0; base <= nbrk; base += 32) {  // lane per window
          const int q = base + lane;
          double dl[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
          float lo = 0.f, hi = 0.f;
          if (q <= nbrk) hi = q < nbrk ? R[8 * q] : 1.f;
          if (q > 0 && q <= nbrk) {  // coordinate q - 1 has left
            const float* o = R + 8 * (q - 1);
            lo = o[0];
            const double xj = o[1], dj = o[2], uj = o[3], vj = o[4], bj = o[5], hjj = o[6];
            dl[0] = (xj * hjj - 2.0 * uj) * xj;
            dl[1] = xj * dj * hjj - xj * vj - dj * uj;
            dl[2] = (dj * hjj - 2.0 * vj) * dj;
            dl[3] = -bj * xj;
            dl[4] = -bj * dj;
          }
          if (nbrk > 0)
#pragma unroll
            for (int k = 0; k < 5; ++k)
              for (int o = 1; o < 32; o <<= 1) {
                const double e = __shfl_up_sync(dense::FULL, dl[k], o);
                if (lane >= o) dl[k] += e;
              }
#pragma unroll
          for (int k = 0; k < 5; ++k) {
            const double all = __shfl_sync(dense::FULL, dl[k], 31);
            dl[k] += c5[k];
            c5[k] += all;
          }
          double bc = 1e300;
          float ba = 0.f;
          if (q <= nbrk && hi - lo > 1.0e-7f) {
            const double c0 = 0.5 * dl[0] + dl[3], c1 = dl[1] + dl[4], c2 = dl[2];
            const float opt = c2 > 0.0 ? fminf(fmaxf((float)(-c1 / c2), lo), hi) : 0.5f * (lo + hi);
            const float cand[3] = {lo, hi, opt};
            for (int k = 0; k < 3; ++k) {
              const double al = cand[k];
              const double cost = c0 + c1 * al + 0.5 * c2 * al * al;
              if (cost < bc) { bc = cost; ba = cand[k]; }
            }
          }
          for (int o = 1; o < 32; o <<= 1) {  // the least cost, of equal ones the first window's
            const double oc = __shfl_down_sync(dense::FULL, bc, o);
            const float oa = __shfl_down_sync(dense::FULL, ba, o);
            if (lane + o < 32 && oc < bc) { bc = oc; ba = oa; }
          }
          bc = __shfl_sync(dense::FULL, bc, 0);
          ba = __shfl_sync(dense::FULL, ba, 0);
          if (bc < best_c) { best_c = bc; best_a = ba; }
        }
        if (lane == 0) flag[7] = (best_a <= 0.f || cur - best_c <= 1.0e-7 * (1.0 + fabs(cur))) ? 0.f : best_a;
      }
      __syncthreads();
      const float best_a = flag[7];
      if (best_a <= 0.f) break;
      const float xn = x + best_a * d;
      x = in ? (xn < 0.f ? 0.f : xn) : 0.f;
      done = it + 1;
    }
    if (done == max_it) status |= NEWT_WS_ITER_CAP;
  }
  __syncthreads();
  if (in) {
    X[r] = x;
    wf[L.con + CF * sccon[ord[r >> 2]] + C_IMP + (r & 3)] = x;
  }
  __syncthreads();
  // the bodies' velocity changes M^-1 J^T f (world frame): a thread per body
  // and component, the rows in order
  for (int e = tid; e < 6 * nb; e += ROWS) {
    const int b = e / 6, c = e % 6;
    const int o = c < 3 ? c : c + 1;
    float s = 0.f;
    for (int k = 0; k < nact; ++k) {
      const int bb = bod[k], sa = (bb & 0xffff) == b, sb = bb >> 16 == b;
      if (!sa && !sb) continue;
      const float* rr = sc0 + (size_t)SC * ord[k] + S_ROWS + 16 + (sa ? 0 : 8) + o;
#pragma unroll
      for (int q = 0; q < 4; ++q) s += rr[32 * q] * X[4 * k + q];
    }
    (c < 3 ? wf[L.dv + 3 * b + c] : wf[L.dw + 3 * b + c - 3]) = s;
  }
  if (tid == 0 && status)
    atomicOr(reinterpret_cast<unsigned*>(g.I + (size_t)w * g.lay.istride + g.lay.status), status);
}

// Every world of the table: those of up to `small` rows (NB_SMALL or none) are
// solved here, the larger ones listed.
__global__ void __launch_bounds__(NB_SMALL, 12) pile_k_newton_small(const PileGroupDev* G, const int* wseg, int ng,
                                                                    int total, int small, NewtonLists lists) {
  extern __shared__ __align__(16) float nbs[];
  const int t = blockIdx.x;
  const int gi = find_seg(wseg, ng, t);
  const PileGroupDev& g = G[gi];
  if (g.solve != PS_NEWTON) return;
  const int w = t - wseg[gi];
  if (w >= g.n || !g.I[(size_t)w * g.lay.istride + g.lay.live]) return;
  const WsLay L = ws_layout(g.nb, g.np, g.maxc);
  const int nact = active_contacts(L, reinterpret_cast<const int*>(g.scr + (size_t)w * g.sstride + L.nf));
  if (nact == 0) return;  // the velocity changes stay zero
  const int c = newton_class(4 * nact, small);
  if (c >= 0) {
    if (threadIdx.x == 0) lists.items[c * lists.stride + atomicAdd(lists.counts + c, 1)] = t;
    return;
  }
  newton_block<NB_SMALL>(g, w, nbs);
}
template <int ROWS, int BLOCKS>
__global__ void __launch_bounds__(ROWS, BLOCKS) pile_k_newton_block(const PileGroupDev* G, const int* wseg, int ng,
                                                                    NewtonLists lists) {
  extern __shared__ __align__(16) float nbs[];
  const int c = ROWS == NB_MID ? 0 : 1, n = lists.counts[c];
  for (int k = blockIdx.x; k < n; k += gridDim.x) {
    const int t = lists.items[c * lists.stride + k];
    const int gi = find_seg(wseg, ng, t);
    newton_block<ROWS>(G[gi], t - wseg[gi], nbs);
    __syncthreads();
  }
}

}  // namespace

// Floats of one world's Newton region (past its pile scratch).
extern "C" size_t newt_pile_newton_bytes(int maxc) { return (size_t)newton_layout(maxc).words * sizeof(float); }

// Kernel attributes for the shared memory (outside stream capture).
extern "C" cudaError_t newt_pile_newton_prepare() {
  const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
  const cudaError_t e =
      cudaFuncSetAttribute(pile_k_newton_block<NB_MID, 3>, attr, (int)(nb_smem(NB_MID).words * sizeof(float)));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(pile_k_newton_block<NB_BIG, 1>, attr, (int)(nb_smem(NB_BIG).words * sizeof(float)));
}

// The dense Newton solve (the solo step's and the contact sensors' re-solve).
// The lists of larger worlds lie in the island lists, which no Newton step
// reads, their counters at the end of the island counters' (zeroed with them).
// The grids of the listed worlds fill the chip once.  Returns the launches.
extern "C" int newt_launch_pile_newton_solve(const PileGroupDev* dG, const int* dwseg, int ng, int total_worlds,
                                             int* lists, int slots, int* counters, cudaStream_t st) {
  if (total_worlds <= 0) return 0;
  static const int sms = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 152;
  }();
  const NewtonLists nl{lists, counters, slots};
  auto grid = [&](int per) { return total_worlds < per * sms ? total_worlds : per * sms; };
  auto bytes = [](int rows) { return nb_smem(rows).words * sizeof(float); };
  // Worlds that the second instance takes in one wave anyway wait for nothing
  // there: 250 worlds of 10 boxes took 38 us here for the smallest, then 78 us
  // for the rest; all together they take the 78.
  const int small = total_worlds <= 3 * sms ? 0 : NB_SMALL;
  pile_k_newton_small<<<total_worlds, NB_SMALL, bytes(NB_SMALL), st>>>(dG, dwseg, ng, total_worlds, small, nl);
  pile_k_newton_block<NB_MID, 3><<<grid(3), NB_MID, bytes(NB_MID), st>>>(dG, dwseg, ng, nl);
  pile_k_newton_block<NB_BIG, 1><<<grid(1), NB_BIG, bytes(NB_BIG), st>>>(dG, dwseg, ng, nl);
  pile_k_newton_warp<<<grid(16), 32, 0, st>>>(dG, dwseg, ng, nl);
  return 4;
}
