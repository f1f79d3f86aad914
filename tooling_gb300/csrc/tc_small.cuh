// The tree-contact solve of trees of up to 24 DoF whose rows are facets or
// normals (included by newton_kernels.cu): the same stages as tc_rows_solve,
// a warp per world and a lane per row, for worlds of up to 32 rows; a world
// with more takes tc_rows_solve itself.
//
// What bounds it: instruction supply.  One warp per block with the stages in
// a straight line (tc_k_solve) waits 6.5 of every 14.4 cycles an instruction
// for the instruction itself, since no two warps of an SM are at the same
// place; so a block's worlds pass the stages together, and the stages are
// arranged for few instructions:
//   * joint axes and levers are rotated once per link, the rows and the link
//     Jacobians read them from shared memory;
//   * M's entries go row by row of its lower triangle, so the base's entries,
//     which sum every link, share their round;
//   * the two factors (M + dt B and M) take a half-warp each, two rows a
//     lane, four columns a load;
//   * the rows' forward substitution and the inverse weights' (of the links
//     that own rows) share one pass, a lane per right-hand side;
//   * the Newton system stays in a lane's registers, and the sums that steer
//     its line search are reduced together.
// Measured on 16384 quadrupeds (13 links, 18 DoF, 0 to 28 rows; GB300, a
// launch): 1737 us as tc_k_solve, 32000 instructions a world at 14.4 cycles
// each; 413 us here, 11200 at 10.3 (fetch waits 0.4).  Four, eight or sixteen
// worlds a block differ by 1 %, 0 and 6 %.
//
// Quotients by a factor's pivots are x * r corrected by the remainder
// x - q d (r the correctly rounded reciprocal of d; P. Markstein, IBM J. Res.
// Dev. 34(1), 1990).

constexpr int TCS_WARPS = 8;  // worlds (warps) per block
constexpr int TCS_ROWS = 32;  // rows of a world, a lane each
constexpr int TCS_LDH = 36;   // row stride of H: float4 loads of eight rows meet no bank twice

namespace {

// Row stride of the mass matrix and of Y: a multiple of four, odd in float4s.
NEWT_HD int tcs_ld(int nv) { return 4 * (((nv + 3) / 4) | 1); }

struct TcsSmem { int topo, arms, wa, qd, lm, ldm, di, links, s2, over, jv, iw, jt, y, h, x, words; };
NEWT_HD TcsSmem tcs_smem(int L, int nv, int maxc, int rpc) {
  const TcSmem o = tc_smem(L, nv, maxc, rpc);
  const int ld = tcs_ld(nv);
  TcsSmem m;
  int f = o.vec;  // the row map and the link poses are tc_smem's
  m.topo = f; f += up4(L);
  m.arms = f; f += up4(9 * L);
  m.wa = f; f += up4(3 * nv);
  m.qd = f; f += 2 * up4(nv);
  m.lm = f; f += nv * ld;   // M + dt B, then its factor; row-major
  m.ldm = f; f += nv * ld;  // M
  m.di = f; f += 2 * 24;    // reciprocals of the pivots
  m.links = f; f += up4(L);
  m.s2 = f; f += up4(3 * L);
  m.over = f;
  // the link Jacobians and inertias, until M is summed
  m.jv = f;
  m.iw = f + 3 * nv * L;
  const int a = 3 * nv * L + 7 * L;
  // then Y and the right-hand sides, and H in their place
  m.y = f;
  m.h = f + TCS_ROWS * ld;
  m.jt = m.h;
  const int jt = nv * 32, hh = TCS_ROWS * TCS_LDH;
  m.x = m.h + (jt > hh ? jt : hh);
  const int b = m.x + 2 * TCS_ROWS - f;
  f += up4(a > b ? a : b);
  m.words = f > o.words ? f : o.words;  // tc_rows_solve's own layout lies in the same words
  return m;
}

NEWT_D float4 f4(const float* p) { return *reinterpret_cast<const float4*>(p); }
// x / d with r = 1 / d
NEWT_D float quot(float x, float d, float r) {
  const float q = x * r;
  return fmaf(fmaf(-q, d, x), r, q);
}

// Columns of the point Jacobian, as chain_columns, from the levers of
// tc_kinematics and the angular axes `wa` of the DoFs.
template <class F>
NEWT_D void arm_columns(const float* pose, const int* topo, const float* arms, const float* wa, int l, V3 pt, F col) {
  V3 d = pt - ldv3(pose + 7 * l);
  for (int i = l;;) {
    const int t = topo[i], jt = t >> 8 & 255, vo = t >> 16;
    if (i == 0) {
      if (jt == JF)
        for (int k = 0; k < 3; ++k) {
          const V3 aw = ldv3(wa + 3 * (vo + k));
          col(vo + k, cross(aw, d));
          col(vo + 3 + k, aw);
        }
      break;
    }
    const float* ar = arms + 9 * i;
    const V3 aw = ldv3(ar);
    if (jt == JH) col(vo, cross(aw, d - ldv3(ar + 3)));
    else if (jt == JS) col(vo, aw);
    d = d + ldv3(ar + 6);
    i = topo_parent(t);
  }
}

// Lower Cholesky factors of two n x n row-major matrices, in place (the upper
// triangles stay), n <= 32: half-warp h factors m[h], lane r of it rows r and
// r + 16.  The entries' products are subtracted in column order.  di: 1 / pivot,
// n (<= 24) per matrix.  False when a pivot is not positive.
NEWT_D bool chol_pair(float* m0, float* m1, int n, int ld, float* di, int lane) {
  float* m = lane & 16 ? m1 : m0;
  float* d = di + (lane & 16 ? 24 : 0);
  const int i1 = lane & 15, i2 = i1 + 16;
  float* r1 = m + (i1 < n ? i1 : n - 1) * ld;
  float* r2 = m + (i2 < n ? i2 : n - 1) * ld;
  bool ok = true;
  for (int j = 0; j < n; ++j) {
    const float* rj = m + j * ld;
    float s1 = r1[j], s2 = r2[j];
    for (int k = 0; k < j; k += 4) {
      float4 c = f4(rj + k);
      const float4 a = f4(r1 + k), b = f4(r2 + k);
      if (k + 1 >= j) c.y = 0.f;
      if (k + 2 >= j) c.z = 0.f;
      if (k + 3 >= j) c.w = 0.f;
      s1 = fmaf(-a.x, c.x, s1); s2 = fmaf(-b.x, c.x, s2);
      s1 = fmaf(-a.y, c.y, s1); s2 = fmaf(-b.y, c.y, s2);
      s1 = fmaf(-a.z, c.z, s1); s2 = fmaf(-b.z, c.z, s2);
      s1 = fmaf(-a.w, c.w, s1); s2 = fmaf(-b.w, c.w, s2);
    }
    const float piv = __shfl_sync(FULL, j < 16 ? s1 : s2, (lane & 16) | (j & 15));
    ok = ok && piv > 0.f;
    const float l = sqrtf(piv), inv = 1.f / l;
    if (i1 >= j && i1 < n) r1[j] = i1 == j ? l : s1 * inv;
    if (i2 >= j && i2 < n) r2[j] = i2 == j ? l : s2 * inv;
    if (i1 == 0) d[j] = inv;
    __syncwarp();
  }
  return __all_sync(FULL, ok);
}

// The same of one matrix, a lane per row; the pivots' range.
NEWT_D bool chol_one(float* m, int n, int ld, int lane, float* mn, float* mx) {
  float* r = m + (lane < n ? lane : n - 1) * ld;
  float lo = 1e30f, hi = 0.f;
  bool ok = true;
  for (int j = 0; j < n; ++j) {
    const float* rj = m + j * ld;
    float s = rj[lane < n ? lane : n - 1];  // the upper triangle: column j from row j down
    for (int k = 0; k < j; k += 4) {
      float4 c = f4(rj + k);
      const float4 a = f4(r + k);
      if (k + 1 >= j) c.y = 0.f;
      if (k + 2 >= j) c.z = 0.f;
      if (k + 3 >= j) c.w = 0.f;
      s = fmaf(-a.x, c.x, s);
      s = fmaf(-a.y, c.y, s);
      s = fmaf(-a.z, c.z, s);
      s = fmaf(-a.w, c.w, s);
    }
    const float piv = __shfl_sync(FULL, s, j);
    ok = ok && piv > 0.f;
    const float l = sqrtf(piv), inv = 1.f / l;
    lo = l < lo ? l : lo;
    hi = l > hi ? l : hi;
    if (lane >= j && lane < n) r[j] = lane == j ? l : s * inv;
    __syncwarp();
  }
  *mn = lo;
  *mx = hi;
  return ok;
}

// a / b by Newton steps on the reciprocal from its FP32 value (an FP64 divide
// keeps the FP64 pipe busy several times as long).
NEWT_D double quot_d(double a, double b) {
  const float bf = (float)b;
  if (!(bf > 1e-30f && bf < 1e30f)) return a / b;
  double r = (double)(1.f / bf);
  r = fma(fma(-b, r, 1.0), r, r);
  const double q = a * r;
  return fma(fma(-q, b, a), r, q);
}

// Row times a shared vector (zeros from nr up to the next multiple of four).
NEWT_D float row_dot(const float (&h)[TCS_ROWS], const float* x, int nr) {
  float s = 0.f;
#pragma unroll
  for (int c = 0; c < TCS_ROWS; c += 4)
    if (c < nr) {
      const float4 v = f4(x + c);
      s = fmaf(h[c], v.x, s);
      s = fmaf(h[c + 1], v.y, s);
      s = fmaf(h[c + 2], v.z, s);
      s = fmaf(h[c + 3], v.w, s);
    }
  return s;
}

// dense::newton_solve for nr <= 32 rows, a lane per row.  H: full symmetric
// rows of stride TCS_LDH with zeros up to a multiple of four columns; its
// lower triangle and diagonal are overwritten by the factor.  b: the lane's
// bias; xs: two shared vectors of 32.  Returns the iterations, or -1 (nothing
// solved) when the factor is too ill-conditioned for FP32.  The lane's impulse
// in *x_out, its diagonal entry in *hd_out.
NEWT_D int small_newton(float* H, int nr, float b, float* xs, int iters, int lane, float* x_out, float* hd_out,
                        uint32_t* status) {
  const bool in = lane < nr;
  float* row = H + (in ? lane : nr - 1) * TCS_LDH;
  float h[TCS_ROWS];
#pragma unroll
  for (int c = 0; c < TCS_ROWS; c += 4) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < nr) v = f4(row + c);
    h[c] = v.x; h[c + 1] = v.y; h[c + 2] = v.z; h[c + 3] = v.w;
  }
  const float hd = row[in ? lane : nr - 1];
  __syncwarp();
  float mn, mx;
  *hd_out = hd;
  if (!chol_one(H, nr, TCS_LDH, lane, &mn, &mx) || (mx / mn) * (mx / mn) > 1.0e6f) return -1;
  const float ld = in ? row[lane] : 1.f, li = 1.f / ld;
  float x = 0.f;
  double cur = 0.0;
  int done = 0;
  const int max_it = iters > 1 ? iters : 1;
  float* ps = xs;
  float* ss = xs + TCS_ROWS;
  for (int it = 0; it < max_it; ++it) {
    float hx = 0.f;
    if (it > 0) {
      ps[lane] = x;
      __syncwarp();
      hx = row_dot(h, ps, nr);
      if (!in) hx = 0.f;
    }
    const float grad = in ? hx + b : 0.f;
    // d = -(L L^T)^-1 grad
    float d = -grad;
    for (int k0 = 0; k0 < nr; k0 += 4) {
      const float4 l = f4(row + k0);
      const float lk[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int k = k0 + u;
        const float q = quot(d, ld, li);
        const float y = __shfl_sync(FULL, q, k & 31);
        d = lane > k ? fmaf(-lk[u], y, d) : (lane == k ? q : d);
      }
    }
    if (!in) d = 0.f;
    for (int k = nr - 1; k >= 0; --k) {
      const float l = H[k * TCS_LDH + lane];  // L[k][lane], used below the diagonal
      const float q = quot(d, ld, li);
      const float z = __shfl_sync(FULL, q, k);
      d = lane < k ? fmaf(-l, z, d) : (lane == k ? q : d);
    }
    if (dense::warp_sum(grad * d) >= 0.f) break;
    // ---- exact line search over the projected path (newton.rs:435-556) ----
    const bool fr = x > 0.f || (x == 0.f && d > 0.f);
    float p = fr ? x : 0.f, s = fr ? d : 0.f;
    float brk = (x > 0.f && d < 0.f) ? -x / d : 2.f;
    brk = (brk > 0.f && brk < 1.f) ? brk : 2.f;
    __syncwarp();
    ss[lane] = s;
    if (it > 0) ps[lane] = p;
    __syncwarp();
    float v = row_dot(h, ss, nr), u = it > 0 ? row_dot(h, ps, nr) : 0.f;
    if (!in) { v = 0.f; u = 0.f; }
    double Pu = 0.0, Pv = 0.0, Sv, bP = 0.0, bS;
    if (it == 0) {  // x = 0: p = 0
      double t[2] = {(double)s * (double)v, (double)b * (double)s};
      dense::warp_sums(t, lane);
      Sv = t[0];
      bS = t[1];
    } else {
      double t[8] = {(double)p * (double)u, (double)p * (double)v, (double)s * (double)v, (double)b * (double)p,
                     (double)b * (double)s, (double)x * (double)hx, (double)x * (double)b, 0.0};
      dense::warp_sums(t, lane);
      Pu = t[0]; Pv = t[1]; Sv = t[2]; bP = t[3]; bS = t[4];
      cur = 0.5 * t[5] + t[6];
    }
    float best_a = 0.f, lo = 0.f;
    double best_c = cur;
    for (int guard = 0; guard <= nr; ++guard) {
      const unsigned bm = __reduce_min_sync(FULL, __float_as_uint(brk));  // positive floats order as their bits
      const bool last = !(__uint_as_float(bm) < 2.f);
      const float hi = last ? 1.f : __uint_as_float(bm);
      if (hi - lo > 1.0e-7f) {
        const double c0 = 0.5 * Pu + bP, c1 = Pv + bS, c2 = Sv;
        const float opt = c2 > 0.0 ? fminf(fmaxf((float)quot_d(-c1, c2), lo), hi) : 0.5f * (lo + hi);
        // the candidates lo, hi, opt in order, a lane each
        const float cand = lane == 0 ? lo : lane == 1 ? hi : opt;
        const double a = cand;
        const double cost = c0 + c1 * a + 0.5 * c2 * a * a;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const double ck = __shfl_sync(FULL, cost, k);
          if (ck < best_c) { best_c = ck; best_a = k == 0 ? lo : k == 1 ? hi : opt; }
        }
      }
      if (last) break;
      // coordinate bi leaves the free set: P, S lose it, H P and H S a column
      const int bi = __ffs(__ballot_sync(FULL, __float_as_uint(brk) == bm)) - 1;
      const float xf = __shfl_sync(FULL, p, bi), df = __shfl_sync(FULL, s, bi);
      const double xj = xf, dj = df, uj = __shfl_sync(FULL, u, bi), vj = __shfl_sync(FULL, v, bi),
                   bj = __shfl_sync(FULL, b, bi), hjj = __shfl_sync(FULL, hd, bi);
      Pu += (xj * hjj - 2.0 * uj) * xj;
      Pv += xj * dj * hjj - xj * vj - dj * uj;
      Sv += (dj * hjj - 2.0 * vj) * dj;
      bP -= bj * xj;
      bS -= bj * dj;
      // column bi of H: its upper triangle, both ways
      const float hc = lane == bi ? hd : H[(lane < bi ? lane : bi) * TCS_LDH + (lane < bi ? bi : lane)];
      if (in) {
        u -= xf * hc;
        v -= df * hc;
      }
      if (lane == bi) { p = 0.f; s = 0.f; brk = 2.f; }
      lo = hi;
    }
    if (best_a <= 0.f || cur - best_c <= 1.0e-7 * (1.0 + fabs(cur))) break;
    const float xn = x + best_a * d;
    x = in ? (xn < 0.f ? 0.f : xn) : 0.f;
    done = it + 1;
    __syncwarp();
  }
  if (done == max_it) *status |= NEWT_WS_ITER_CAP;
  *x_out = x;
  return done;
}

// A world of more rows, and the Newton solve with its FP64 factor, out of line.
__device__ __noinline__ void rows_solve_any(const TcGroupDev& G, int w, float* sv, int nr, int ncon, uint32_t status,
                                            int lane) {
  tc_rows_solve<false>(G, w, sv, nr, ncon, status, lane);
}
// H's upper triangle (diagonal hd, a lane's) goes to Hg; its words then hold the vectors.
__device__ __noinline__ int newton_any(float* H, float hd, int nr, float* Hg, float* LH, double* LHd, int ld, float b,
                                       int iters, bool zero_mu, int lane, float* x_out, uint32_t* status) {
  __syncwarp();
  if (lane < nr)
    for (int c = 0; c < nr; ++c)
      Hg[(size_t)c * ld + lane] = c == lane ? hd : H[min(c, lane) * TCS_LDH + max(c, lane)];
  __syncwarp();
  float* v = H;
  v[lane] = 0.f;
  v[32 + lane] = b;
  __syncwarp();
  const int done = dense::newton_solve(Hg, nr, ld, LH, ld, LHd, v, v + 32, v + 64, v + 96, v + 128, v + 160, v + 192,
                                       v + 224, v + 256, iters, zero_mu, lane, status);
  *x_out = lane < nr ? v[lane] : 0.f;
  return done;
}

}  // namespace

__global__ void __launch_bounds__(32 * TCS_WARPS, 2) tc_k_small(const __grid_constant__ TcGroupDev G) {
  extern __shared__ __align__(16) float tcs[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = blockIdx.x * (blockDim.x >> 5) + warp;
  const TreeGroupDev& g = G.t;
  const int cap = g.cap, L = g.L, nv = g.nv;
  const TcLay lay = tc_layout(L, nv, G.ng, G.maxc, G.rpc);
  const TcSmem so = tc_smem(L, nv, G.maxc, G.rpc);
  const TcsSmem sm = tcs_smem(L, nv, G.maxc, G.rpc);
  const int ldm = tcs_ld(nv), nq = up4(nv);
  float* wf = G.scr + (size_t)w * G.sstride;
  float* sv = tcs + (size_t)warp * sm.words;
  float* pose = sv + so.pose;
  int* rcon = reinterpret_cast<int*>(sv + so.rmap);
  int* rfac = rcon + so.ldr;
  int* topo = reinterpret_cast<int*>(sv + sm.topo);
  float* arms = sv + sm.arms;
  float* wa = sv + sm.wa;
  float* qd = sv + sm.qd;
  float* qa = qd + nq;
  float* LM = sv + sm.lm;   // M + dt B, its factor (response, qacc)
  float* LD = sv + sm.ldm;  // M, its factor (diagApprox)
  float* di = sv + sm.di;
  float* Y = sv + sm.y;
  float* H = sv + sm.h;
  float* xs = sv + sm.x;
  const float* con = wf + lay.con;
  uint32_t status = 0;
  int ncon = 0, nr = 0;
  const bool live = w < g.n && g.live[w];  // uniform per warp, as every condition on it below
  float dt = 0.f;
  bool rk4 = false;

  // ---- forward kinematics, joint axes and levers ----
  if (live) {
    dt = g.dtg[w];
    rk4 = g.integ && g.integ[w] == NEWT_INTEGRATOR_RK4;
    if (lane < nv) {
      qd[lane] = g.qd[lane * cap + w];
      qa[lane] = g.qacc[lane * cap + w];
    }
    tc_kinematics(g, w, pose, topo, arms, lane);
    for (int i = lane; i < L; i += 32) {
      const int t = topo[i], jt = t >> 8 & 255, vo = t >> 16;
      if (jt == JF) {
        const Q4 o = Q4{pose[7 * i + 3], pose[7 * i + 4], pose[7 * i + 5], pose[7 * i + 6]};
        for (int k = 0; k < 3; ++k) {
          stv3(wa + 3 * (vo + k), qrot(o, v3(k == 0 ? 1.f : 0.f, k == 1 ? 1.f : 0.f, k == 2 ? 1.f : 0.f)));
          stv3(wa + 3 * (vo + 3 + k), v3(0.f, 0.f, 0.f));
        }
      } else if (jt == JH) {
        stv3(wa + 3 * vo, ldv3(arms + 9 * i));
      } else if (jt == JS) {
        stv3(wa + 3 * vo, v3(0.f, 0.f, 0.f));
      }
    }
    __syncwarp();
  }
  __syncthreads();

  // ---- contacts and their rows ----
  if (live) {
    nr = tc_contacts(G, w, pose, rcon, rfac, false, lane, &ncon, &status);
    __syncwarp();
    if (nr == 0 && lane == 0 && status) atomicOr(g.status + w, status);  // qacc stays a_free
  }
  bool on = nr > 0 && nr <= TCS_ROWS;
  __syncthreads();

  // ---- link COM Jacobians, world inertias and masses, lane per link; M ----
  if (on) {
    float* JV = sv + sm.jv;
    float* IW = sv + sm.iw;  // 6 per link, then the link masses
    float* MS = IW + 6 * L;
    for (int k = 4 * lane; k < 2 * nv * ldm; k += 128)
      *reinterpret_cast<float4*>(LM + k) = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int l = lane; l < L; l += 32) {
      const float* pl = pose + 7 * l;
      float* jv = JV + 3 * nv * l;
      arm_columns(pose, topo, arms, wa, l, ldv3(pl), [&](int k, V3 tr) { stv3(jv + 3 * k, tr); });
      const M3 R = quat_mat(Q4{pl[3], pl[4], pl[5], pl[6]});
      M3 RT;
      for (int r = 0; r < 3; ++r) for (int c = 0; c < 3; ++c) RT.m[r][c] = R.m[c][r];
      const S3 Ib{g.inert[(6 * l) * cap + w], g.inert[(6 * l + 1) * cap + w], g.inert[(6 * l + 2) * cap + w],
                  g.inert[(6 * l + 3) * cap + w], g.inert[(6 * l + 4) * cap + w], g.inert[(6 * l + 5) * cap + w]};
      const S3 Iw = sym_congr(RT, Ib);  // R I R^T
      float* iw = IW + 6 * l;
      iw[0] = Iw.xx; iw[1] = Iw.yy; iw[2] = Iw.zz; iw[3] = Iw.xy; iw[4] = Iw.xz; iw[5] = Iw.yz;
      MS[l] = g.mass[l * cap + w];
    }
    __syncwarp();
    // entry (i, j), i >= j, sums the links below DoF i's joint when DoF j's
    // link is an ancestor of it, in link order, and is zero otherwise
    const int* dmask = G.gtopo + 3 * G.ng;  // subtree masks (lo, hi) per link
    const int* dlink = dmask + 2 * L;       // link of each DoF
    auto subtree = [&](int a) {
      return ((unsigned long long)(unsigned)dmask[2 * a + 1] << 32) | (unsigned)dmask[2 * a];
    };
    for (int i = 0, j = lane;; j += 32) {
      while (i < nv && j > i) j -= ++i;
      if (i >= nv) break;
      const int ai = dlink[i], aj = dlink[j];
      float s = 0.f;
      if ((subtree(aj) >> ai) & 1ull) {
        const V3 wi = ldv3(wa + 3 * i), wj = ldv3(wa + 3 * j);
        for (unsigned long long m = subtree(ai); m; m &= m - 1ull) {
          const int l = __ffsll((long long)m) - 1;
          const float* jv = JV + 3 * nv * l;
          const float* iw = IW + 6 * l;
          const S3 I{iw[0], iw[1], iw[2], iw[3], iw[4], iw[5]};
          s += MS[l] * dot(ldv3(jv + 3 * i), ldv3(jv + 3 * j)) + dot(wi, smv(I, wj));
        }
      }
      // armature (child joints) and, under Euler, the implicit damping dt*B
      // (tree.rs:645-684); RK4 factors M itself (solver.rs:2852-2855)
      float sm_ = s;
      if (i == j) {
        const int jt = topo[ai] >> 8 & 255;
        const float damp = rk4 ? 0.f : dt * g.damp[ai * cap + w];
        if (jt == JF) {
          sm_ = s + damp;
        } else {
          const float arm = g.arm[ai * cap + w];
          sm_ = s + (arm + damp);
          s += arm;
        }
      }
      LD[i * ldm + j] = s;
      LM[i * ldm + j] = sm_;
    }
    __syncwarp();
  }
  __syncthreads();
  if (on) {
    if (!chol_pair(LM, LD, nv, ldm, di, lane)) {
      if (lane == 0) atomicOr(g.status + w, status | NEWT_WS_NOT_PD);
      on = false;
    }
  }
  __syncthreads();

  // ---- rows and links' inverse weights: right-hand sides, their forward
  //      substitutions; A = Y^T Y; regulariser, diagonal and bias ----
  float bias = 0.f, reg = 0.f, mu = 0.f;
  bool facet = false;
  if (on) {
    int* links = reinterpret_cast<int*>(sv + sm.links);
    float* s2 = sv + sm.s2;
    float* Jt = sv + sm.jt;
    for (int l = lane; l < L; l += 32) links[l] = 0;
    __syncwarp();
    const bool row = lane < nr;
    const float* cc = con + CREC * (row ? rcon[lane] : 0);
    const int link = row ? __float_as_int(cc[K_LINK]) : 0, link2 = row ? __float_as_int(cc[K_LINK2]) : -1;
    if (row) {
      links[link] = 1;
      if (link2 >= 0) links[link2] = 1;
    }
    __syncwarp();
    int nl = 0;  // the links that own rows, listed in place
    for (int base = 0; base < L; base += 32) {
      const int l = base + lane;
      const bool has = l < L && links[l];
      const unsigned m = __ballot_sync(FULL, has);
      if (has) links[nl + __popc(m & ((1u << lane) - 1u))] = l;
      nl += __popc(m);
      __syncwarp();
    }
    float vel = 0.f, vfree = 0.f;
    for (int t0 = 0; t0 < nr + 3 * nl; t0 += 32) {
      const int t = t0 + lane, q = t - nr, wl = q >= 0 && q < 3 * nl ? links[q / 3] : 0, axis = q >= 0 ? q % 3 : 0;
      if (t < nr + 3 * nl) {
        // a row: its direction's translational columns (world_jacobian_for_side,
        // solver.rs:3537-3598); a weight: an axis of the link's COM
        int l = wl;
        V3 pt = ldv3(pose + 7 * wl), dir = v3(axis == 0 ? 1.f : 0.f, axis == 1 ? 1.f : 0.f, axis == 2 ? 1.f : 0.f);
        float sign = 1.f;
        if (q < 0) {
          l = link;
          pt = ldv3(cc + K_POS);
          dir = row_direction(cc, rfac[lane]);
          sign = cc[K_SIGN];
        }
        for (int k = 0; k < nv; ++k) Jt[32 * k + lane] = 0.f;
        arm_columns(pose, topo, arms, wa, l, pt, [&](int k, V3 tr) { Jt[32 * k + lane] = dot(tr, dir) * sign; });
        if (q < 0 && link2 >= 0)  // side b of an in-tree pair
          arm_columns(pose, topo, arms, wa, link2, pt, [&](int k, V3 tr) { Jt[32 * k + lane] -= dot(tr, dir); });
        if (q < 0 && rk4)
          for (int k = 0; k < nv; ++k) wf[lay.j0 + (size_t)k * lay.ld + lane] = Jt[32 * k + lane];
      }
      __syncwarp();
      const float* F = q < 0 ? LM : LD;
      const float* fd = q < 0 ? di : di + 24;
      float y[REFINE_NV], ss = 0.f;
#pragma unroll
      for (int k = 0; k < REFINE_NV; ++k) {
        y[k] = 0.f;
        if (k < nv) {
          float s = Jt[32 * k + lane];
          if (t0 == 0) {
            vel += s * qd[k];
            vfree += s * qa[k];
          }
          float dk = 1.f;
#pragma unroll
          for (int m = 0; m <= k; m += 4) {
            const float4 f = f4(F + k * ldm + m);
            if (m < k) s = fmaf(-f.x, y[m], s); else dk = f.x;
            if (m + 1 < k) s = fmaf(-f.y, y[m + 1], s); else if (m + 1 == k) dk = f.y;
            if (m + 2 < k) s = fmaf(-f.z, y[m + 2], s); else if (m + 2 == k) dk = f.z;
            if (m + 3 < k) s = fmaf(-f.w, y[m + 3], s); else if (m + 3 == k) dk = f.w;
          }
          y[k] = quot(s, dk, fd[k]);
          ss += y[k] * y[k];
        }
      }
      if (t < nr) {
#pragma unroll
        for (int k = 0; k < REFINE_NV; k += 4)
          if (k < nv)
            *reinterpret_cast<float4*>(Y + lane * ldm + k) = make_float4(y[k], y[k + 1], y[k + 2], y[k + 3]);
      } else if (q < 3 * nl) {
        s2[3 * wl + axis] = ss;  // |L_D^-1 jv_axis|^2 = jv_axis^T M^-1 jv_axis
      }
      __syncwarp();
    }
    // A, its lower triangle's entries over the lanes
    for (int r = 0, c = lane;; c += 32) {
      while (r < nr && c > r) c -= ++r;
      if (r >= nr) break;
      float s = 0.f;
      for (int k = 0; k < nv; k += 4) {
        const float4 a = f4(Y + r * ldm + k), b = f4(Y + c * ldm + k);
        s = fmaf(a.x, b.x, s);
        s = fmaf(a.y, b.y, s);
        s = fmaf(a.z, b.z, s);
        s = fmaf(a.w, b.w, s);
      }
      H[r * TCS_LDH + c] = s;
      H[c * TCS_LDH + r] = s;
    }
    if (row)
      for (int c = nr; c < up4(nr); ++c) H[lane * TCS_LDH + c] = 0.f;
    // regulariser and bias (solver.rs:3068-3121), the inverse weights of
    // tree_body_invweight0 and tree_contact_diag_approx
    if (row) {
      const float pen = cc[K_PEN] - cc[K_GAP];
      mu = cc[K_MU];
      const Soft s{cc[K_SR], cc[K_SR + 1], cc[K_SI], cc[K_SI + 1], cc[K_SI + 2], cc[K_SI + 3], (int)cc[K_SI + 4]};
      const float d = impedance_at(-pen, s);
      facet = rfac[lane] >= 0;
      float twl = ((s2[3 * link] + s2[3 * link + 1]) + s2[3 * link + 2]) / 3.f;
      if (link2 >= 0) twl += ((s2[3 * link2] + s2[3 * link2 + 1]) + s2[3 * link2 + 2]) / 3.f;
      const float base = (1.f - d) / d * (facet ? twl * (1.f + mu * mu) : twl);
      reg = facet ? 2.f * mu * mu * base : base;
      // the position term drives the facets and the normal row only
      const float position = (facet || rfac[lane] == R_NORMAL) ? -pen : 0.f;
      const float free_dv = __fmul_rn(vfree, dt);  // J . (a_free dt)
      bias = free_dv - reference_accel(position, vel, s.tc, s.dr, s, dt) * dt;
    }
    __syncwarp();
  }
  __syncthreads();

  // ---- impulses ----
  float x = 0.f;
  int done = 0;
  if (on) {
    const int iters = G.iters[w];
    const bool row = lane < nr;
    if (G.mode[w] == NEWT_SOLVER_PGS) {
      // dense Gauss-Seidel (world_pgs_non_negative, solver.rs:3851-3862)
      const float diag = row ? H[lane * TCS_LDH + lane] + reg : 1.f;
      for (int it = 0; it < iters; ++it)
        for (int r = 0; r < nr; ++r) {
          const float s = dense::warp_sum(row ? H[r * TCS_LDH + lane] * x : 0.f);
          const float p = x - ((bias + s) + reg * x) / diag;
          if (lane == r) x = p < 0.f ? 0.f : p;
        }
      done = iters;
    } else {
      if (row) H[lane * TCS_LDH + lane] += reg;
      __syncwarp();
      float hd;
      done = small_newton(H, nr, bias, xs, iters, lane, &x, &hd, &status);
      if (done < 0)  // zero-friction facets duplicate rows: newt's solver-only pivot (solver.rs:3215-3232)
        done = newton_any(H, hd, nr, wf + lay.H, wf + lay.LH, reinterpret_cast<double*>(wf + lay.LHd), lay.ld, bias,
                          iters, __any_sync(FULL, facet && mu == 0.f), lane, &x, &status);
    }
  } else if (nr > TCS_ROWS) {
    rows_solve_any(G, w, sv, nr, ncon, status, lane);
  }
  __syncthreads();

  // ---- outputs: impulses, J^T f / dt, qacc = a_free + (M + dt B)^-1 J^T f / dt ----
  // J^T = L Y, so (L L^T)^-1 J^T f / dt = L^-T (Y f) / dt: one back
  // substitution.  RK4 worlds hold J^T f / dt over the integrator's stages.
  if (on) {
    if (lane < nr) wf[lay.imp + lane] = x;
    xs[lane] = x;
    __syncwarp();
    const int kv = lane < nv ? lane : nv - 1;
    float v = 0.f, jf = 0.f;
    for (int r = 0; r < nr; ++r) v += Y[r * ldm + kv] * xs[r];
    v = v / dt;
    if (rk4 && lane < nv) {
      for (int r = 0; r < nr; ++r) jf += wf[lay.j0 + (size_t)lane * lay.ld + r] * xs[r];
      g.cfrc[(size_t)w * g.cstride + lane] = jf / dt;
    }
    const float dv = LM[kv * ldm + kv], rv = di[kv];
    for (int k = nv - 1; k >= 0; --k) {
      const float f = LM[k * ldm + kv];
      const float q = quot(v, dv, rv);
      const float z = __shfl_sync(FULL, q, k);
      v = lane < k ? fmaf(-f, z, v) : (lane == k ? q : v);
    }
    if (lane < nv) g.qacc[lane * cap + w] = qa[lane] + v;
    if (lane == 0) {
      wf[lay.misc + 2] = __int_as_float(done);
      if (status) atomicOr(g.status + w, status);
    }
  }
}
