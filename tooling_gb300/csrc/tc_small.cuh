// The tree-contact solve of trees of up to 24 DoF whose rows are facets or
// normals (included by newton_kernels.cu): the same stages as tc_rows_solve,
// a warp per world and a lane per row, for worlds of up to 32 rows; the
// worlds with more take tc_rows_solve, in a launch of their own (tc_k_listed)
// or, where a block is one world, here.
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
//     lane; every factor and substitution advances four columns at a time,
//     the 4 x 4 blocks by every lane for itself;
//   * the rows' forward substitution and the inverse weights' (of the links
//     that own rows) share one pass, a lane per right-hand side;
//   * the Newton system stays in a lane's registers, and the sums that steer
//     its line search are reduced together.
// Measured on 16384 quadrupeds (13 links, 18 DoF, 0 to 28 rows; GB300, a
// launch): 1737 us as tc_k_solve, 32000 instructions a world at 14.4 cycles
// each; 376 us here, 10400 at 10.2 (fetch waits 1.0, global memory 1.8, shared
// memory 1.1, barriers 1.0).  Blocks of four worlds, four to an SM, against
// eight and two: 917 and 939 us for two env-steps; without the barriers around
// the Newton stage 932 to 948.

constexpr int TCS_WARPS = 4;   // worlds (warps) per block
constexpr int TCS_BLOCKS = 4;  // blocks per SM
constexpr int TCS_FEW = 8;     // worlds per SM up to which each has a block of its own
constexpr int TCS_MANY = 64;   // worlds per SM from which a few large ones are solved in their blocks
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
  m.lm = f; f += up4(nv) * ld;   // M + dt B, then its factor; row-major
  m.ldm = f; f += up4(nv) * ld;  // M
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
  const int b = m.x + 3 * TCS_ROWS - f;
  f += up4(a > b ? a : b);
  m.words = f > o.words ? f : o.words;  // tc_rows_solve's own layout lies in the same words
  return m;
}

NEWT_D float4 f4(const float* p) { return *reinterpret_cast<const float4*>(p); }

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

// The 4 x 4 diagonal block of a factor, and its reciprocal pivots.
struct Block4 {
  float l00, l10, l11, l20, l21, l22, l30, l31, l32, l33, i0, i1, i2, i3;
  // of the block whose lower entries row q's lane holds in s[0..q]; q's lane is `lane0` + q
  NEWT_D bool factor(const float (&s)[4], int lane0) {
    auto at = [&](int u, int q) { return __shfl_sync(FULL, s[u], lane0 + q); };
    const float d00 = at(0, 0), d10 = at(0, 1), d20 = at(0, 2), d30 = at(0, 3), d11 = at(1, 1), d21 = at(1, 2),
                d31 = at(1, 3), d22 = at(2, 2), d32 = at(2, 3), d33 = at(3, 3);
    l00 = sqrtf(d00); i0 = 1.f / l00;
    l10 = d10 * i0; l20 = d20 * i0; l30 = d30 * i0;
    const float e11 = fmaf(-l10, l10, d11);
    l11 = sqrtf(e11); i1 = 1.f / l11;
    l21 = fmaf(-l20, l10, d21) * i1; l31 = fmaf(-l30, l10, d31) * i1;
    const float e22 = fmaf(-l21, l21, fmaf(-l20, l20, d22));
    l22 = sqrtf(e22); i2 = 1.f / l22;
    l32 = fmaf(-l31, l21, fmaf(-l30, l20, d32)) * i2;
    const float e33 = fmaf(-l32, l32, fmaf(-l31, l31, fmaf(-l30, l30, d33)));
    l33 = sqrtf(e33); i3 = 1.f / l33;
    return d00 > 0.f && e11 > 0.f && e22 > 0.f && e33 > 0.f;
  }
  // of the factor m (row-major) at row p, reciprocals at di + p
  NEWT_D void load(const float* m, int ld, int p, const float* di) {
    const float4 r1 = f4(m + (p + 1) * ld + p), r2 = f4(m + (p + 2) * ld + p), r3 = f4(m + (p + 3) * ld + p),
                 i = f4(di + p);
    l00 = m[p * ld + p];
    l10 = r1.x; l11 = r1.y;
    l20 = r2.x; l21 = r2.y; l22 = r2.z;
    l30 = r3.x; l31 = r3.y; l32 = r3.z; l33 = r3.w;
    i0 = i.x; i1 = i.y; i2 = i.z; i3 = i.w;
  }
  // row q of the block, zeros above the diagonal; its reciprocal pivot
  NEWT_D float4 row(int q) const {
    return make_float4(q == 0 ? l00 : q == 1 ? l10 : q == 2 ? l20 : l30, q == 0 ? 0.f : q == 1 ? l11 : q == 2 ? l21 : l31,
                       q < 2 ? 0.f : q == 2 ? l22 : l32, q < 3 ? 0.f : l33);
  }
  NEWT_D float inv(int q) const { return q == 0 ? i0 : q == 1 ? i1 : q == 2 ? i2 : i3; }
  // a row below the block
  NEWT_D float4 below(const float (&s)[4]) const {
    const float y0 = s[0] * i0, y1 = fmaf(-y0, l10, s[1]) * i1, y2 = fmaf(-y1, l21, fmaf(-y0, l20, s[2])) * i2;
    return make_float4(y0, y1, y2, fmaf(-y2, l32, fmaf(-y1, l31, fmaf(-y0, l30, s[3]))) * i3);
  }
  // L y = v and L^T z = v
  NEWT_D float4 forward(float4 v) const {
    const float y0 = quot(v.x, l00, i0), y1 = quot(fmaf(-l10, y0, v.y), l11, i1);
    const float y2 = quot(fmaf(-l21, y1, fmaf(-l20, y0, v.z)), l22, i2);
    return make_float4(y0, y1, y2, quot(fmaf(-l32, y2, fmaf(-l31, y1, fmaf(-l30, y0, v.w))), l33, i3));
  }
  NEWT_D float4 backward(float4 v) const {
    const float z3 = quot(v.w, l33, i3), z2 = quot(fmaf(-l32, z3, v.z), l22, i2);
    const float z1 = quot(fmaf(-l21, z2, fmaf(-l31, z3, v.y)), l11, i1);
    return make_float4(quot(fmaf(-l10, z1, fmaf(-l20, z2, fmaf(-l30, z3, v.x))), l00, i0), z1, z2, z3);
  }
};
NEWT_D float pick(float4 v, int q) { return q == 0 ? v.x : q == 1 ? v.y : q == 2 ? v.z : v.w; }
NEWT_D float4 shfl4(float v, int lane0) {
  return make_float4(__shfl_sync(FULL, v, lane0), __shfl_sync(FULL, v, lane0 + 1), __shfl_sync(FULL, v, lane0 + 2),
                     __shfl_sync(FULL, v, lane0 + 3));
}
NEWT_D float minus4(float s, float4 a, float4 b) {  // s - a . b, in order
  return fmaf(-a.w, b.w, fmaf(-a.z, b.z, fmaf(-a.y, b.y, fmaf(-a.x, b.x, s))));
}

// Lower Cholesky factors of two n x n row-major matrices (n a multiple of
// four, <= 24; zeros above the diagonal), in place, four columns at a time:
// half-warp h factors m[h], lane r of it rows r and r + 16.  The entries'
// products are subtracted in column order.  di: 1 / pivot, 24 per matrix.
// False when a pivot is not positive.
NEWT_D bool chol_pair(float* m0, float* m1, int n, int ld, float* di, int lane) {
  float* m = lane & 16 ? m1 : m0;
  float* d = di + (lane & 16 ? 24 : 0);
  const int i1 = lane & 15, i2 = i1 + 16;
  float* r1 = m + (i1 < n ? i1 : n - 1) * ld;
  float* r2 = m + (i2 < n ? i2 : n - 1) * ld;
  bool ok = true;
  for (int p = 0; p < n; p += 4) {
    const float4 c1 = f4(r1 + p), c2 = f4(r2 + p);
    float s1[4] = {c1.x, c1.y, c1.z, c1.w}, s2[4] = {c2.x, c2.y, c2.z, c2.w};
    for (int k = 0; k < p; k += 4) {
      const float4 a = f4(r1 + k), b = f4(r2 + k);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float4 c = f4(m + (p + u) * ld + k);
        s1[u] = minus4(s1[u], a, c);
        s2[u] = minus4(s2[u], b, c);
      }
    }
    Block4 B;
    ok = (p < 16 ? B.factor(s1, (lane & 16) | p) : B.factor(s2, (lane & 16) | (p & 15))) && ok;
    if (i1 >= p && i1 < n) *reinterpret_cast<float4*>(r1 + p) = i1 < p + 4 ? B.row(i1 - p) : B.below(s1);
    if (i2 >= p && i2 < n) *reinterpret_cast<float4*>(r2 + p) = i2 < p + 4 ? B.row(i2 - p) : B.below(s2);
    if (i1 < 4) d[p + i1] = B.inv(i1);
    __syncwarp();
  }
  return __all_sync(FULL, ok);
}

// The same of one matrix, a lane per row, the entries taken above the
// diagonal, which stay; the range of the first nr pivots.
NEWT_D bool chol_one(float* m, int n, int nr, int ld, float* di, int lane, float* mn, float* mx) {
  const int i = lane < n ? lane : n - 1;
  float* r = m + i * ld;
  float lo = 1e30f, hi = 0.f;
  bool ok = true;
  for (int p = 0; p < n; p += 4) {
    float s[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) s[u] = m[(p + u) * ld + i];
    for (int k = 0; k < p; k += 4) {
      const float4 a = f4(r + k);
#pragma unroll
      for (int u = 0; u < 4; ++u) s[u] = minus4(s[u], a, f4(m + (p + u) * ld + k));
    }
    Block4 B;
    ok = B.factor(s, p) && ok;
    lo = fminf(lo, B.l00);
    hi = fmaxf(hi, B.l00);
    if (p + 1 < nr) { lo = fminf(lo, B.l11); hi = fmaxf(hi, B.l11); }
    if (p + 2 < nr) { lo = fminf(lo, B.l22); hi = fmaxf(hi, B.l22); }
    if (p + 3 < nr) { lo = fminf(lo, B.l33); hi = fmaxf(hi, B.l33); }
    __syncwarp();
    if (lane >= p + 4 && lane < n) {
      *reinterpret_cast<float4*>(r + p) = B.below(s);
    } else if (lane >= p && lane < n) {
      const float4 v = B.row(lane - p);
      r[p] = v.x;
      if (lane > p) r[p + 1] = v.y;
      if (lane > p + 1) r[p + 2] = v.z;
      if (lane > p + 2) r[p + 3] = v.w;
      di[lane] = B.inv(lane - p);
    }
    __syncwarp();
  }
  *mn = lo;
  *mx = hi;
  return ok;
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
// bias; xs: two shared vectors of 32, then the factor's 32 reciprocal pivots.  Returns the iterations, or -1 (nothing
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
  const int n = up4(nr);
  float* di = xs + 2 * TCS_ROWS;
  __syncwarp();
  if (lane >= nr && lane < n)  // rows of the identity up to a multiple of four
    for (int c = lane; c < n; ++c) H[lane * TCS_LDH + c] = c == lane ? 1.f : 0.f;
  __syncwarp();
  float mn, mx;
  *hd_out = hd;
  if (!chol_one(H, n, nr, TCS_LDH, di, lane, &mn, &mx) || (mx / mn) * (mx / mn) > 1.0e6f) return -1;
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
    for (int p = 0; p < n; p += 4) {
      Block4 B;
      B.load(H, TCS_LDH, p, di);
      const float4 y = B.forward(shfl4(d, p));
      d = lane >= p + 4 ? minus4(d, f4(row + p), y) : lane >= p ? pick(y, lane - p) : d;
    }
    if (!in) d = 0.f;
    for (int p = n - 4; p >= 0; p -= 4) {
      Block4 B;
      B.load(H, TCS_LDH, p, di);
      const float* c = H + p * TCS_LDH + lane;  // below the diagonal: the factor's columns, by rows
      const float l3 = c[3 * TCS_LDH], l2 = c[2 * TCS_LDH], l1 = c[TCS_LDH], l0 = c[0];
      const float4 z = B.backward(shfl4(d, p));
      d = lane < p ? fmaf(-l0, z.x, fmaf(-l1, z.y, fmaf(-l2, z.z, fmaf(-l3, z.w, d)))) : lane < p + 4 ? pick(z, lane - p) : d;
    }
    if (!in) d = 0.f;
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
        double c0 = 0.0, c1 = bS;
        const double c2 = Sv;
        if (it > 0) {
          c0 = 0.5 * Pu + bP;
          c1 += Pv;
        }
        auto take = [&](float a) {
          const double cost = c0 + c1 * (double)a + 0.5 * c2 * (double)a * (double)a;
          if (cost < best_c) { best_c = cost; best_a = a; }
        };
        if (c2 > 0.0) {  // the ends are no lower than the clamped minimiser
          take(fminf(fmaxf(quot_d(-c1, c2), lo), hi));
        } else {
          take(lo);
          take(hi);
          take(0.5f * (lo + hi));
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

// A world of more rows where the launch lists none, and the Newton solve with
// its FP64 factor, out of line.
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

__global__ void __launch_bounds__(32 * TCS_WARPS, TCS_BLOCKS) tc_k_small(const __grid_constant__ TcGroupDev G) {
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
  bool rk4 = false, here = false;

  // ---- forward kinematics, joint axes and levers ----
  PairGeoms first;
  if (live) {
    first = tc_pair(G, w, lane);
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
    nr = tc_contacts(G, w, pose, first, rcon, rfac, false, lane, &ncon, &status);
    __syncwarp();
    if (nr > TCS_ROWS && !G.list) {  // a block of one warp
      rows_solve_any(G, w, sv, nr, ncon, status, lane);
      return;
    }
    if (nr > TCS_ROWS) {
      int before = 0;
      if (lane == 0 && G.here > 0) before = atomicAdd(G.list + 2, 1);
      here = __shfl_sync(FULL, before, 0) < G.here;
      if (!here && lane == 0) G.list[3 + atomicAdd(G.list, 1)] = w;
    }
    if ((nr == 0 || (nr > TCS_ROWS && !here)) && lane == 0 && status) atomicOr(g.status + w, status);
  }
  bool on = nr > 0 && nr <= TCS_ROWS;  // without rows qacc stays a_free
  if (!__syncthreads_or(on || here)) return;

  // ---- link COM Jacobians, world inertias and masses, lane per link; M ----
  if (on) {
    float* JV = sv + sm.jv;
    float* IW = sv + sm.iw;  // 6 per link, then the link masses
    float* MS = IW + 6 * L;
    for (int k = 4 * lane; k < 2 * nq * ldm; k += 128)
      *reinterpret_cast<float4*>(LM + k) = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncwarp();
    if (lane < nq - nv)  // the identity up to a multiple of four rows
      LM[(nv + lane) * (ldm + 1)] = LD[(nv + lane) * (ldm + 1)] = 1.f;
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
    if (!chol_pair(LM, LD, nq, ldm, di, lane)) {
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
  } else if (here) {
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
    if (lane >= nv) v = 0.f;
    for (int p = nq - 4; p >= 0; p -= 4) {
      Block4 B;
      B.load(LM, ldm, p, di);
      const float* c = LM + p * ldm + min(lane, nq - 1);
      const float l3 = c[3 * ldm], l2 = c[2 * ldm], l1 = c[ldm], l0 = c[0];
      const float4 z = B.backward(shfl4(v, p));
      v = lane < p ? fmaf(-l0, z.x, fmaf(-l1, z.y, fmaf(-l2, z.z, fmaf(-l3, z.w, v)))) : lane < p + 4 ? pick(z, lane - p) : v;
    }
    if (lane < nv) g.qacc[lane * cap + w] = qa[lane] + v;
    if (lane == 0) {
      wf[lay.misc + 2] = __int_as_float(done);
      if (status) atomicOr(g.status + w, status);
    }
  }
}
