// The batched form's free-body step: two launches per env-step over every
// pile world of a size class.
//
//   pile_k_contacts  warp per world: the world record to shared memory;
//                    AABBs, sorted sweep, ordered pair list and narrowphase
//                    (pile_collide.cuh); the active contacts in contact
//                    order, their dependency levels, and a lane per contact
//                    for its row constants, written in sweep order
//   pile_k_sweep     32, 16 or 8 lanes per world: the row constants to shared
//                    memory once, then the PGS sweeps over the levels (the
//                    contacts of one level touch disjoint bodies), two lanes
//                    per contact, and the integration (semi-implicit Euler or
//                    RK4) into the world record
//
// What bounds it.  A contact's update waits on the previous update of its
// bodies: a settled 16-body pile takes 50 sweeps of about five levels in
// series, whatever runs beside it, and a warp alone issues an instruction
// every three to four cycles.  So what counts is how many instructions one
// level takes and how many worlds share them.
//
// Restates, for FP32 on sm_103a:
//   newt/src/world.rs:1459-1537   World::step phase order (Euler branch)
//   newt/src/solver.rs:703-1257   solve_free_bodies_diag_mode, PGS branch: rows,
//                                 regularisation, bias (:752-1061) and the
//                                 sweeps (:1085-1200)
//   newt/src/solver.rs:1448-1518  pgs_step_non_negative, pgs_step_pyramidal_pair
//   newt/src/solver.rs:1892-2036  row_body_diagonal, row_residual,
//                                 apply_impulse_delta
//   newt/src/solver.rs:3401-3429  pyramidal facet rows n +- mu t
//   newt/src/world.rs:3104-3112   tangent_basis
//
// Gauss-Seidel order.  newt sweeps each island's contacts in contact order.
// A contact update reads the velocity accumulators of its (at most two)
// dynamic bodies, which only earlier contacts on the same bodies have
// changed; running the levels in order therefore reproduces the serial sweep
// of every island exactly (islands never share a body).
//
// Contact update.  A pyramidal contact has four facet rows r = n + s_r mu
// t_q(r) (s = +, -, +, -; q = 1, 1, 2, 2).  Three dot products with the
// bodies' velocity changes (J_n, mu J_t1, mu J_t2) give the four residuals;
// newt's row steps run in registers -- the non-negative step on row 0, then
// the pyramidal pairs (0,1) and (2,3) -- advancing the residuals by the exact
// row-space block A_rs = J_r M^-1 J_s^T after every step (what re-reading
// J_r . v gives, up to rounding), and the summed impulse changes are applied
// to the bodies once.
//
// Scaled velocities.  With M^-1 = C C^T (sqrt(1/m) and R C_b, C_b the Cholesky
// factor of the body-frame inverse inertia) the sweeps carry u with v = C u
// and rows J C: the same six floats per side and row read the velocity and
// change it, where J and M^-1 J^T would be twelve.  A lane holds one side of
// a contact; two packed multiply-adds (f32x2) make each three of a row's six
// products, and one shuffle adds the sides.
//
// Measured (GB300, us an env-step, one warp per world for the whole horizon
// before -> now): ten worlds of 16 bodies 206 -> 88, 8192 of 16 bodies
// 1100 -> 493, 700 of 53 bodies 790 -> 247, 1500 of 12 capsules (RK4)
// 196 -> 96.
#include <algorithm>
#include <cmath>
#include <cstddef>

#include "../../include/newt_gpu.h"
#include "pile_solver.cuh"

using namespace pile;

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int N_BUCKET = 256; // cost classes of the queue sort

// One contact's row constants and impulses.
struct Side { float n[6], t1[6], t2[6], pad[2]; };  // J C of the normal and mu times the tangents: linear, angular
struct alignas(16) Row {
  Side side[2];              // zero for a static side
  float f[4], b[4], id[4];   // impulses, biases, inverse row diagonals
  float a00, a10, a20, a30;  // A (a00 with the regulariser): column 0,
  float a21, a31, a32, reg;  // and what the later rows take
  float p0[3], p1[3], pad[2];  // the pairs' h11, h01, h00 (newt's row diagonals and A_ij) over their determinants
};
constexpr int ROW_V4 = sizeof(Row) / 16;
constexpr int ROW_F4 = offsetof(Row, f) / 16;
static_assert(sizeof(Side) % 16 == 0 && offsetof(Row, f) % 16 == 0, "rows move as float4");
static_assert(ROW_V4 % 2 == 1, "lanes on different rows read shared memory without bank conflicts");
static_assert(4 * ROW_V4 <= SC, "a row fits the solver record's slot");
// A row's bodies (nb: a static side) and which pairs have a determinant that
// is not positive: a | b << 8 | pairs << 16.

// Contacts as pile_k_contacts holds them (shared memory, the ones past its
// capacity in the scratch record): point, normal, depth, friction, then the
// geoms and the entities as 16-bit pairs.
enum { K_POS = 0, K_N = 3, K_PEN = 6, K_MU = 7, K_GEOM = 8, K_ENT = 9, K_WORDS = 11 };  // odd: no bank conflicts

// C_b with C_b C_b^T = the body-frame inverse inertia (lower Cholesky factor;
// a pivot lost to rounding is zero).
NEWT_D M3 inverse_inertia_factor(const S3& I) {
  const float a = sqrtf(fmaxf(I.xx, 0.f)), ia = a > 0.f ? 1.f / a : 0.f;
  const float b = I.xy * ia, c = I.xz * ia;
  const float d = sqrtf(fmaxf(I.yy - b * b, 0.f)), id = d > 0.f ? 1.f / d : 0.f;
  const float e = (I.yz - b * c) * id;
  return M3{{{a, 0.f, 0.f}, {b, d, 0.f}, {c, e, sqrtf(fmaxf(I.zz - c * c - e * e, 0.f))}}};
}

// newt's facet rows of one active contact (newt/src/solver.rs:752-1061).
// `L.iinvw`: per body R C_b (nine floats).  Returns the row's bodies word.
NEWT_D int row_assemble(const WsLay& L, const float* wf, const float* cf, Row& R) {
  const int nb = L.nb;
  const float dt = wf[L.dtg];
  const V3 grav = v3(wf[L.dtg + 1], wf[L.dtg + 2], wf[L.dtg + 3]);
  const float* soft = wf + L.soft;
  float tc = soft[0], dr = soft[1];
  const bool direct = tc < 0.f;
  if (!direct && tc < 2.f * dt) tc = 2.f * dt;  // safe_solref (solver.rs:331-338)
  const float dmax = fminf(fmaxf(soft[3], 1.0e-4f), 0.9999f);
  const int ent = __float_as_int(cf[K_ENT]), ea = ent & 0xffff, eb = ent >> 16;
  const float pen = cf[K_PEN], mu = cf[K_MU];
  const V3 n = ld3(cf + K_N), pos = ld3(cf + K_POS);
  V3 ref = fabsf(n.z) < 0.9f ? v3(0.f, 0.f, 1.f) : v3(1.f, 0.f, 0.f);
  V3 t1 = cross(ref, n);
  const float tl = sqrtf(len2(t1));
  t1 = tl == 0.f ? v3(0.f, 0.f, 0.f) : t1 * (1.f / tl);
  const V3 t2 = cross(n, t1);
  // per side: rows J C, the points' velocity, the inverse mass
  float im[2];
  V3 ang[2][3];
  V3 rel = v3(0.f, 0.f, 0.f);
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int e = k ? eb : ea;
    const bool dyn = e < nb;
    const float sg = k ? -1.f : 1.f;
    im[k] = dyn ? 1.f / wf[L.mass + e] : 0.f;
    const float s = sqrtf(im[k]) * sg;
    const V3 arm = dyn ? pos - ld3(wf + L.pos + 3 * e) : v3(0.f, 0.f, 0.f);
    M3 C = {};
    if (dyn) {
      const float* m = wf + L.iinvw + 9 * e;
      for (int q = 0; q < 9; ++q) C.m[q / 3][q % 3] = m[q];
    }
    ang[k][0] = mtv(C, cross(arm, n)) * sg;
    ang[k][1] = mtv(C, cross(arm, t1)) * sg;
    ang[k][2] = mtv(C, cross(arm, t2)) * sg;
    auto put = [](float* o, V3 l, V3 a) { o[0] = l.x; o[1] = l.y; o[2] = l.z; o[3] = a.x; o[4] = a.y; o[5] = a.z; };
    put(R.side[k].n, n * s, ang[k][0]);
    put(R.side[k].t1, t1 * (s * mu), ang[k][1] * mu);
    put(R.side[k].t2, t2 * (s * mu), ang[k][2] * mu);
    R.side[k].pad[0] = R.side[k].pad[1] = 0.f;
    if (dyn)
      rel = rel + (ld3(wf + L.vel + 3 * e) + cross(qrot(ld4(wf + L.quat + 4 * e), ld3(wf + L.omg + 3 * e)), arm)) * sg;
  }
  const float tran = im[0] + im[1];
  const float d = impedance(-pen, soft);
  const float reg = d > 0.f ? 2.f * mu * mu * ((1.f - d) / d * (tran * (1.f + mu * mu))) : 0.f;
  float b_, k0;
  if (direct) { b_ = -dr / dmax; k0 = -soft[0] / (dmax * dmax); }
  else { b_ = 2.f / (dmax * tc); k0 = d / (dmax * dmax * tc * tc * dr * dr); }
  // gravity moves both sides of a contact of two bodies alike
  const float gs = (ea < nb ? 1.f : 0.f) - (eb < nb ? 1.f : 0.f);
  const V3 ds[3] = {n, t1, t2};
  V3 dir[4], ra[4], rb[4];
  float diag[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int q = r < 2 ? 1 : 2;
    const float s = (r & 1) ? -mu : mu;
    dir[r] = n + ds[q] * s;
    ra[r] = ang[0][0] + ang[0][q] * s;
    rb[r] = ang[1][0] + ang[1][q] * s;
    diag[r] = ((len2(ra[r]) + im[0]) + (len2(rb[r]) + im[1])) + reg;  // row_body_diagonal
    const float aref = -b_ * dot(rel, dir[r]) - k0 * (-pen);
    R.b[r] = gs * dot(grav * dt, dir[r]) - aref * dt;
    R.id[r] = 1.f / diag[r];
    R.f[r] = 0.f;
  }
  // exact row-space block A_rs = J_r M^-1 J_s^T
  auto arow = [&](int r, int s) { return dot(dir[r], dir[s]) * tran + (dot(ra[r], ra[s]) + dot(rb[r], rb[s])); };
  R.reg = reg;
  R.a00 = arow(0, 0) + reg; R.a10 = arow(0, 1); R.a20 = arow(0, 2); R.a30 = arow(0, 3);
  R.a21 = arow(1, 2); R.a31 = arow(1, 3); R.a32 = arow(2, 3);
  // pyramidal pair blocks (solver.rs:1037-1061)
  int single = 0;
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const float off = p ? R.a32 : R.a10, det = diag[2 * p] * diag[2 * p + 1] - off * off;
    const float idet = det > 0.f ? 1.f / det : 0.f;
    if (!(det > 0.f)) single |= 1 << p;
    float* o = p ? R.p1 : R.p0;
    o[0] = diag[2 * p + 1] * idet;
    o[1] = off * idet;
    o[2] = diag[2 * p] * idet;
  }
  R.pad[0] = R.pad[1] = 0.f;
  return (ea < nb ? ea : nb) | (eb < nb ? eb : nb) << 8 | single << 16;
}

// ---- packed pairs of floats ----
typedef unsigned long long f32x2;
NEWT_D f32x2 pack2(float a, float b) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
NEWT_D float sum2(f32x2 v) { float a, b; asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); return a + b; }
NEWT_D f32x2 mul2(f32x2 a, f32x2 b) { f32x2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
NEWT_D f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
NEWT_D f32x2 lo2(float4 v) { return pack2(v.x, v.y); }
NEWT_D f32x2 hi2(float4 v) { return pack2(v.z, v.w); }

// newt's pyramidal pair step (RowStep::pair, solver.rs:1476-1518), its four
// cases chosen by selects: both impulses non-negative, the pair; one
// negative, it is zero and the other steps alone; both, zero.  h11, h01, h00:
// the pair's block over its determinant.
NEWT_D void pair_step(float fi, float fj, float ri, float rj, float h11, float h01, float h00, float idi, float idj,
                      float* ni, float* nj) {
  const float ui = fmaf(h01, rj, fmaf(-h11, ri, fi)), uj = fmaf(h01, ri, fmaf(-h00, rj, fj));
  const float si = fmaxf(fmaf(-ri, idi, fi), 0.f), sj = fmaxf(fmaf(-rj, idj, fj), 0.f);
  *ni = ui >= 0.f ? (uj >= 0.f ? ui : si) : 0.f;
  *nj = uj >= 0.f ? (ui >= 0.f ? uj : sj) : 0.f;
}

constexpr int FARS = 10;  // percent of a warp's rows past their place that pile_k_sweep's own loops put up with
constexpr int ACC = 12;  // floats per body of the accumulators (six used): 16-byte aligned, spread over the banks

// What a contact's update reads of its row and does not change.
struct RowRegs { float4 q0, q1, q2, q3, q4, b, id, a0, a1, pa, pb; };
NEWT_D RowRegs row_load(const float4* x, int stride, int side) {
  const float4* sx = x + side * (5 * stride);
  const float4* cx = x + 10 * stride;
  return RowRegs{sx[0], sx[stride], sx[2 * stride], sx[3 * stride], sx[4 * stride], cx[stride], cx[2 * stride],
                 cx[3 * stride], cx[4 * stride], cx[5 * stride], cx[6 * stride]};
}

// One contact's update (newt/src/solver.rs:1085-1200, 1448-1518) on two
// neighbouring lanes, this one on side `side`; R: the row's constants, fp: its
// impulses; A: its body's accumulator (u linear, angular), `write`: unless the
// side is static.  The other lanes of `pair` take part in the shuffles.
// SINGLE: a pair whose determinant is not positive (a bit of `single`) takes
// two half-line steps.  ahead: called once the accumulator's loads are out.
template <bool SINGLE, class F>
NEWT_D void row_update(const RowRegs& R, float4* fp, float* A, bool write, int single, int side, unsigned pair, F ahead) {
  const float4 u01 = *reinterpret_cast<const float4*>(A);
  const float2 u2 = *reinterpret_cast<const float2*>(A + 4);
  const float4 f = *fp;
  ahead();
  const float4 b = R.b, id = R.id, a0 = R.a0, a1 = R.a1, pa = R.pa, pb = R.pb;
  const f32x2 n0 = lo2(R.q0), n1 = hi2(R.q0), n2 = lo2(R.q1), s0 = hi2(R.q1), s1 = lo2(R.q2), s2 = hi2(R.q2),
              t0 = lo2(R.q3), t1 = hi2(R.q3), t2 = lo2(R.q4);
  f32x2 v0 = lo2(u01), v1 = hi2(u01), v2 = pack2(u2.x, u2.y);
  float dn = sum2(fma2(n2, v2, fma2(n1, v1, mul2(n0, v0))));
  float d1 = sum2(fma2(s2, v2, fma2(s1, v1, mul2(s0, v0))));
  float d2 = sum2(fma2(t2, v2, fma2(t1, v1, mul2(t0, v0))));
  dn += __shfl_xor_sync(pair, dn, 1);
  d1 += __shfl_xor_sync(pair, d1, 1);
  d2 += __shfl_xor_sync(pair, d2, 1);
  // residuals with the row's own regulariser
  float e0 = (fmaf(a1.w, f.x, b.x) + dn) + d1, e1 = (fmaf(a1.w, f.y, b.y) + dn) - d1;
  float e2 = (fmaf(a1.w, f.z, b.z) + dn) + d2, e3 = (fmaf(a1.w, f.w, b.w) + dn) - d2;
  const float m0 = fmaxf(fmaf(-e0, id.x, f.x), 0.f);
  {
    const float g = m0 - f.x;
    e0 = fmaf(a0.x, g, e0); e1 = fmaf(a0.y, g, e1); e2 = fmaf(a0.z, g, e2); e3 = fmaf(a0.w, g, e3);
  }
  float r0, r1, r2, r3;
  pair_step(m0, f.y, e0, e1, pa.x, pa.y, pa.z, id.x, id.y, &r0, &r1);
  if (SINGLE && (single & 1)) {
    r0 = fmaxf(fmaf(-e0, id.x, m0), 0.f);
    r1 = fmaxf(fmaf(-fmaf(a0.y, r0 - m0, e1), id.y, f.y), 0.f);
  }
  {
    const float g0 = r0 - m0, g1 = r1 - f.y;
    e2 = fmaf(a0.z, g0, fmaf(a1.x, g1, e2));
    e3 = fmaf(a0.w, g0, fmaf(a1.y, g1, e3));
  }
  pair_step(f.z, f.w, e2, e3, pa.w, pb.x, pb.y, id.z, id.w, &r2, &r3);
  if (SINGLE && (single & 2)) {
    r2 = fmaxf(fmaf(-e2, id.z, f.z), 0.f);
    r3 = fmaxf(fmaf(-fmaf(a1.z, r2 - f.z, e3), id.w, f.w), 0.f);
  }
  // u += J_n^T sum df + mu J_t1^T (df0 - df1) + mu J_t2^T (df2 - df3)
  const float h0 = r0 - f.x, h1 = r1 - f.y, h2 = r2 - f.z, h3 = r3 - f.w;
  const float Fn = (h0 + h1) + (h2 + h3), F1 = h0 - h1, F2 = h2 - h3;
  const f32x2 gn = pack2(Fn, Fn), g1 = pack2(F1, F1), g2 = pack2(F2, F2);
  v0 = fma2(t0, g2, fma2(s0, g1, fma2(n0, gn, v0)));
  v1 = fma2(t1, g2, fma2(s1, g1, fma2(n1, gn, v1)));
  v2 = fma2(t2, g2, fma2(s2, g1, fma2(n2, gn, v2)));
  if (write) {
    *reinterpret_cast<ulonglong2*>(A) = make_ulonglong2(v0, v1);
    *reinterpret_cast<f32x2*>(A + 4) = v2;
  }
  if (!side) *fp = make_float4(r0, r1, r2, r3);
}

// The same out of line, for rows in either memory and any pairs.
__device__ __noinline__ void row_update_far(float4* x, int stride, float* A, bool write, int single, int side,
                                            unsigned pair) {
  row_update<true>(row_load(x, stride, side), x + ROW_F4 * stride, A, write, single, side, pair, [] {});
}

// The sweeps of a warp whose schedule or more than a few of its rows exceed
// their place in shared memory: rows from either memory, any pairs, the
// schedule from the scratch record.  Out of line, so that pile_k_sweep's own
// loop keeps its registers.  As there, a round's constants are read while the
// one before it updates, its rows' bodies a round before that and its bounds
// one more.  Contacts between boxes come in fours on the same two bodies, so
// stacks and walls have as many rounds: us an env-step with every far row read
// in its own round, and now (one warp per world for the whole horizon in brackets): 1000
// walls of 8 boxes 1203, 643 (849), of 16 2135, 1474 (1544), 8192 of 16 9123,
// 5829 (8382), 1000 stacks of 16 1655, 877 (1187).
// The lane's world: `fit` of its nact rows lie at `mine`, all at `rec`; nr
// rounds that start at loff[], body words `words`, `iters` sweeps; nrm and itm:
// the warp's rounds and sweeps.
struct MixedWorld {
  float4 *zero, *mine, *rec;
  float* acc;
  const int *loff, *words;
  int fit, nact, nr, iters, nb;
};
__device__ __noinline__ void sweep_mixed(const MixedWorld W, int nrm, int itm, int slot, int side) {
  float4 *const zero = W.zero, *const mine = W.mine, *const rec = W.rec;
  float* const acc = W.acc;
  const int *const loff = W.loff, *const words = W.words;
  const int fit = W.fit, nact = W.nact, nr = W.nr, iters = W.iters, nb = W.nb;
  int ra = 0, ia = 0, left = itm * nrm;
  if (left <= 0) return;
  struct Bounds { int lo, hi; };
  auto bounds = [&]() {  // of the next round, none past the end
    Bounds b{0, 0};
    if (ia < iters && ra < nr) b = Bounds{loff[ra], loff[ra + 1]};
    if (++ra == nrm) { ra = 0; ++ia; }
    return b;
  };
  struct Place { int s, word; };  // a row or -1, its bodies
  auto place = [&](Bounds b) {
    Place p{b.lo + slot < b.hi ? b.lo + slot : -1, nb | nb << 8};
    if (p.s >= 0) p.word = words[p.s];
    return p;
  };
  auto row = [&](Place p) { return p.s < 0 ? zero : p.s < fit ? mine + (size_t)p.s * ROW_V4 : rec + p.s; };
  auto stride = [&](Place p) { return p.s >= fit ? nact : 1; };
  auto load = [&](Place p) { return row_load(row(p), stride(p), side); };
  auto update = [&](const RowRegs& R, Place p, auto ahead) {
    const int b = (side ? p.word >> 8 : p.word) & 0xff;
    row_update<true>(R, row(p) + ROW_F4 * stride(p), acc + ACC * b, b < nb, p.s < 0 ? 0 : p.word >> 16, side, FULL, ahead);
    __syncwarp();
  };
  Bounds b2 = bounds();
  Place p0 = place(b2), p1;
  b2 = bounds();
  p1 = place(b2);
  b2 = bounds();
  RowRegs R0 = load(p0), R1;
  Place p2;
  for (; left > 1; left -= 2) {
    update(R0, p0, [&] { R1 = load(p1); p2 = place(b2); b2 = bounds(); });
    p0 = p2;
    update(R1, p1, [&] { R0 = load(p0); p2 = place(b2); b2 = bounds(); });
    p1 = p2;
  }
  if (left > 0) update(R0, p0, [] {});
}

}  // namespace

// ---------------------------------------------------------------------------
// the queue: worlds sorted by last call's cost, most costly first
// ---------------------------------------------------------------------------
// Counting sort by cost class (4 classes per octave of cost); the order
// inside a class is unspecified, which changes which warp steps a world and
// never what it computes.  One block.
__global__ void __launch_bounds__(1024) pile_k_queue_sort(const unsigned* __restrict__ cost, int n,
                                                          int* __restrict__ queue) {
  __shared__ int hist[N_BUCKET];
  auto bucket = [](unsigned c) {
    const float l = log2f((float)c + 1.f) * 4.f;
    const int b = (int)l;
    return b < N_BUCKET ? b : N_BUCKET - 1;
  };
  for (int b = threadIdx.x; b < N_BUCKET; b += blockDim.x) hist[b] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) atomicAdd(&hist[bucket(cost[i])], 1);
  __syncthreads();
  if (threadIdx.x == 0) {  // exclusive starts, most costly class first
    int run = 0;
    for (int b = N_BUCKET - 1; b >= 0; --b) { const int c = hist[b]; hist[b] = run; run += c; }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) queue[atomicAdd(&hist[bucket(cost[i])], 1)] = i;
}

// ---------------------------------------------------------------------------
// pile_k_contacts
// ---------------------------------------------------------------------------
namespace {

// Per-warp shared memory of pile_k_contacts, in words: the world record's
// model and state as they lie there (PileLayout's floats up to the contacts,
// its ints up to the contact pairs), per body R C_b, the AABBs, the pair list,
// then the first `ccap` contacts.  The pair list's
// place holds the active contacts' lists once the narrowphase is done.
struct HotLay {
  WsLay L;  // offsets from the floats and from the ints, as collide() takes them
  int ints, con, ccap, words;
};
NEWT_HD HotLay hot_layout(const PileLayout& P, int nb, int np, int maxc) {
  HotLay h;
  WsLay& L = h.L;
  L = WsLay{};
  L.nb = nb; L.np = np; L.ng = nb + np; L.maxc = maxc;
  const int all = L.ng * (L.ng - 1) / 2;
  L.pcap = all < 2 * maxc ? all : 2 * maxc;
  L.pos = P.pos; L.quat = P.quat; L.vel = P.vel; L.omg = P.omg; L.mass = P.mass; L.iinvb = P.iinv; L.size = P.size;
  L.gpos = P.gpos; L.gquat = P.gquat; L.plane = P.plane; L.fric = P.fric; L.margin = P.margin; L.soft = P.soft;
  L.dtg = P.dtg;
  int f = P.cdata;  // a multiple of 4
  L.iinvw = f; f += 9 * nb; L.aabb = f; f += 6 * L.ng;
  f = (f + 3) / 4 * 4;
  h.ints = f;
  L.shape = P.shape; L.gent = P.gent;
  int i = (P.cpair + 3) / 4 * 4;
  L.misc = i; i += 4;
  const int lists = 2 * L.pcap > 3 * maxc + 2 ? 2 * L.pcap : 3 * maxc + 2;
  L.pairs = i; i += lists;
  f += i;
  h.con = f;
  const int c = 2 * nb + nb / 4 + 8;
  h.ccap = c < maxc ? c : maxc;
  f += K_WORDS * h.ccap;
  h.words = (f + 3) / 4 * 4;
  return h;
}

NEWT_D void copy16(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src));
}
NEWT_D void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// What pile_k_contacts leaves for pile_k_sweep in the world's scratch record:
// the rows at L.sc (float4 q of row s at q * nact + s, in sweep order), their
// body words at L.ci, and these ints.
enum { B_NACT = 0, B_ROUNDS = 1, B_CON = 2, B_RND = 3 };  // at L.misc; B_CON, B_RND: totals over the graph's env-steps

struct Worlds {
  const PileGroupDev* G;
  const int* wseg;
  int ng;
  const int* queue;  // nullable
  int n;
};
// World `item` of the launch, or null (past the end, or not live).
NEWT_D const PileGroupDev* world_at(const Worlds& W, int item, int* w, int* flat) {
  if (item >= W.n) return nullptr;
  const int t = W.queue ? W.queue[item] : item;
  const int gi = find_seg(W.wseg, W.ng, t);
  const PileGroupDev* g = W.G + gi;
  *w = t - W.wseg[gi];
  *flat = t;
  if (*w >= g->n || !g->I[(size_t)*w * g->lay.istride + g->lay.live]) return nullptr;
  return g;
}

}  // namespace

// `cap`: contacts per round of the sweeps; `stride`: words of shared memory
// per warp; `last`: the call's last env-step (the contacts go to the world
// record); `work`: pile_k_sweep's.  (Its counters of levels are added here,
// where the levels are: as totals in pile_k_sweep they cost that loop 5%, by
// its registers.)  The warps of a block meet between the phases: the code is
// long and runs once per world, and warps that are spread over it wait for
// instructions more than for anything else.
__global__ void __launch_bounds__(256, 2) pile_k_contacts(Worlds W, int cap, int stride, int last,
                                                       unsigned long long* work) {
  extern __shared__ __align__(16) float psm[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  int w = 0, flat;
  const PileGroupDev* gp = world_at(W, blockIdx.x * (blockDim.x >> 5) + wib, &w, &flat);
  float* sf = psm + (size_t)wib * stride;
  HotLay H;
  int* si = nullptr;
  if (gp) {
    H = hot_layout(gp->lay, gp->nb, gp->np, gp->maxc);
    si = reinterpret_cast<int*>(sf) + H.ints;
    const float* F = gp->F + (size_t)w * gp->lay.fstride;
    const int* I = gp->I + (size_t)w * gp->lay.istride;
    for (int k = 4 * lane; k < gp->lay.cdata; k += 128) copy16(sf + k, F + k);
    for (int k = 4 * lane; k < gp->lay.cpair; k += 128) copy16(si + k, I + k);
    copies_done();
    __syncwarp();
    const WsLay& L = H.L;
    for (int b = lane; b < L.nb; b += 32) {
      const M3 R = quat_mat(ld4(sf + L.quat + 4 * b)), B = inverse_inertia_factor(lds(sf + L.iinvb + 6 * b));
      float* o = sf + L.iinvw + 9 * b;
      for (int q = 0; q < 9; ++q)
        o[q] = R.m[q / 3][0] * B.m[0][q % 3] + R.m[q / 3][1] * B.m[1][q % 3] + R.m[q / 3][2] * B.m[2][q % 3];
    }
  }
  // the scratch record: contacts past the shared ones, the rows, the schedule
  float* xf = gp ? gp->scr + (size_t)w * gp->sstride : nullptr;
  const int maxc = gp ? gp->maxc : 0;
  WsLay X;
  if (gp) X = ws_layout(gp->nb, gp->np, maxc);
  int* xi = gp ? reinterpret_cast<int*>(xf + X.nf) : nullptr;
  auto contact = [&](int c) { return c < H.ccap ? sf + H.con + K_WORDS * c : xf + X.con + K_WORDS * (c - H.ccap); };
  __syncthreads();
  if (gp)
    collide(H.L, sf, si, lane, [&](int c, V3 pos, V3 n, float pen, float mu, int ga, int gb, int ea, int eb) {
      float* cf = contact(c);
      st3(cf + K_POS, pos); st3(cf + K_N, n);
      cf[K_PEN] = pen; cf[K_MU] = mu;
      cf[K_GEOM] = __int_as_float(ga | gb << 16);
      cf[K_ENT] = __int_as_float(ea | eb << 16);
    });
  __syncthreads();
  int nact = 0;
  unsigned short *act = nullptr, *pos = nullptr;
  if (gp) {
    const WsLay& L = H.L;
    const int nb = L.nb, nc = si[L.misc + 1];
    // active contacts in contact order (solver.rs:762-769): a dynamic side
    // and penetration beyond the gap (gap = 0)
    act = reinterpret_cast<unsigned short*>(si + L.pairs);  // contact of each
    pos = act + maxc;                                       // its place in sweep order
    unsigned short* body = pos + maxc;                      // its bodies (bytes; 255: static)
    short* lev = reinterpret_cast<short*>(body + maxc);     // its level
    short* pa = lev + maxc;                                 // its bodies' last earlier contacts
    short* pb = pa + maxc;
    const unsigned lt = (1u << lane) - 1u;
    for (int c0 = 0; c0 < nc; c0 += 32) {
      const int c = c0 + lane;
      bool on = false;
      int ea = 0, eb = 0;
      if (c < nc) {
        const float* cf = contact(c);
        const int ent = __float_as_int(cf[K_ENT]);
        ea = ent & 0xffff; eb = ent >> 16;
        on = (ea < nb || eb < nb) && cf[K_PEN] > 0.f;
      }
      const unsigned m = __ballot_sync(FULL, on);
      if (on) {
        const int k = nact + __popc(m & lt);
        act[k] = (unsigned short)c;
        body[k] = (unsigned short)((ea < nb ? ea : 255) | (eb < nb ? eb : 255) << 8);
      }
      nact += __popc(m);
    }
    __syncwarp();
    // Levels: a contact's is one more than the highest of the last earlier
    // contacts on its dynamic bodies, so that running the levels in order is
    // the serial sweep.  The last earlier contacts by a scan of the list, the
    // levels by relaxation (a pass settles one level more at least).
#pragma unroll 1
    for (int k = lane; k < nact; k += 32) {
      const int me = body[k], a = me & 255, b = me >> 8;
      int qa = -1, qb = -1;
#pragma unroll 4
      for (int q = 0; q < k; ++q) {
        const int o = body[q], oa = o & 255, ob = o >> 8;
        if (a != 255 && (oa == a || ob == a)) qa = q;
        if (b != 255 && (oa == b || ob == b)) qb = q;
      }
      pa[k] = (short)qa;
      pb[k] = (short)qb;
      lev[k] = 1;
    }
    __syncwarp();
    for (;;) {
      bool up = false;
#pragma unroll 1
      for (int k = lane; k < nact; k += 32) {
        const int qa = pa[k], qb = pb[k];
        const int l = 1 + max(qa >= 0 ? (int)lev[qa] : 0, qb >= 0 ? (int)lev[qb] : 0);
        if (l != lev[k]) { up = true; lev[k] = (short)l; }
      }
      if (!__any_sync(FULL, up)) break;
      __syncwarp();
    }
    // sweep order: by level, rounds of at most `cap` contacts; each round's
    // first row goes to the scratch record's schedule
    int* loff = xi + X.scid;
    int row0 = 0, rounds = 0, levels = 0, eights = 0;
    for (int v = 1; row0 < nact; ++v) {
      int cnt = 0;
#pragma unroll 1
      for (int k0 = 0; k0 < nact; k0 += 32) {
        const int k = k0 + lane;
        const bool in = k < nact && lev[k] == v;
        const unsigned m = __ballot_sync(FULL, in);
        if (in) pos[k] = (unsigned short)(row0 + cnt + __popc(m & lt));
        cnt += __popc(m);
      }
      const int nr = (cnt + cap - 1) / cap;
      if (lane < nr) loff[rounds + lane] = row0 + cap * lane;
      row0 += cnt;
      rounds += nr;
      ++levels;
      eights += (cnt + 7) / 8;
    }
    if (lane == 0) {
      loff[rounds] = nact;
      xi[X.misc + B_NACT] = nact;
      xi[X.misc + B_ROUNDS] = rounds;
      if (levels > 0) {
        atomicAdd(work + 1, (unsigned long long)eights * (unsigned long long)max(si[gp->lay.iters], 0));
        atomicAdd(work + 2, (unsigned long long)levels);
      }
    }
    __syncwarp();
  }
  __syncthreads();
  if (!gp) return;
  const WsLay& L = H.L;
  const PileLayout& P = gp->lay;
  float* F = gp->F + (size_t)w * P.fstride;
  int* I = gp->I + (size_t)w * P.istride;
  // rows, a lane per contact
  float4* rec = reinterpret_cast<float4*>(xf + X.sc);
  int *place = xi + X.sccon, *word = xi + X.ci;
#pragma unroll 1
  for (int k = lane; k < nact; k += 32) {
    union { Row R; float4 v[ROW_V4]; } u;
    const int s = pos[k];
    word[s] = row_assemble(L, sf, contact(act[k]), u.R);
#pragma unroll
    for (int q = 0; q < ROW_V4; ++q) rec[(size_t)q * nact + s] = u.v[q];
    if (last) place[s] = act[k];
  }
  const int nc = si[L.misc + 1];
  if (last) {  // the diagnostics surface (the sweeps add the impulses)
#pragma unroll 1
    for (int c = lane; c < nc; c += 32) {
      const float* cf = contact(c);
      const int gm = __float_as_int(cf[K_GEOM]);
      I[P.cpair + 2 * c] = gm & 0xffff; I[P.cpair + 2 * c + 1] = gm >> 16;
      for (int k = 0; k < 7; ++k) F[P.cdata + 7 * c + k] = cf[k];
      for (int k = 0; k < P.rpc; ++k) F[P.imp + P.rpc * c + k] = 0.f;
    }
    if (lane == 0) I[P.ncon] = nc;
  }
  if (lane == 0 && si[L.misc + 2]) atomicOr(reinterpret_cast<unsigned*>(I + P.status), NEWT_WS_CONTACT_OVERFLOW);
}

// ---------------------------------------------------------------------------
// pile_k_sweep
// ---------------------------------------------------------------------------
// S lanes per world, one warp per block.  Shared memory: per world nbm + 1
// accumulators, then `space` float4: a row of zeros, the schedule (per round
// and lane the row's and the accumulator's byte offsets) and the rows, taken
// in world order (rows past the space stay in the scratch record).  A lane
// without a contact in a round updates the row of zeros against the static
// side's zero: the round is straight-line code, where a branch around it and
// one at each store took a sixth of its time.
// work: [0] active contacts summed over every world's env-steps, [3] worlds
// stepped; pile_k_contacts adds [1] the levels' groups of eight contacts summed
// over the sweeps and [2] the levels summed over env-steps.  cost (per flat
// world index): this graph's rounds over its sweeps plus 64 per contact, the
// sort key of its next replay's queue.  `first`, `tally`: the graph's first and
// last env-step; `last`: the call's last.
NEWT_HD size_t sweep_smem(int S, int nbm, int space) {
  return (size_t)(32 / S) * (nbm + 1) * ACC * 4 + (size_t)space * 16;
}

template <int S>
__global__ void __launch_bounds__(32, 12) pile_k_sweep(Worlds W, int nbm, int space, int first, int tally, int last,
                                                       unsigned long long* work, unsigned* cost) {
  extern __shared__ __align__(16) float4 ssm[];
  constexpr int N = 32 / S;
  const int lane = threadIdx.x, sub = lane / S, l = lane % S, slot = l >> 1, side = l & 1;
  const unsigned pair = 3u << (lane & 30);
  int w = 0, flat = 0;
  const PileGroupDev* g = world_at(W, blockIdx.x * N + sub, &w, &flat);
  float* acc = reinterpret_cast<float*>(ssm) + (size_t)sub * (nbm + 1) * ACC;
  float4* zero = ssm + (size_t)N * (nbm + 1) * ACC / 4;
  if (lane < ROW_V4) zero[lane] = make_float4(0.f, 0.f, 0.f, 0.f);
  int nb = 0, nact = 0, nr = 0, iters = 0;
  float4* rec = nullptr;
  int* xi = nullptr;
  WsLay X;
  if (g) {
    X = ws_layout(g->nb, g->np, g->maxc);
    float* xf = g->scr + (size_t)w * g->sstride;
    xi = reinterpret_cast<int*>(xf + X.nf);
    rec = reinterpret_cast<float4*>(xf + X.sc);
    nb = g->nb;
    nact = xi[X.misc + B_NACT];
    nr = xi[X.misc + B_ROUNDS];
    iters = g->I[(size_t)w * g->lay.istride + g->lay.iters];
  }
  for (int b = l; b < ACC * (nbm + 1); b += S) acc[b] = 0.f;
  int base = 0, rows = 0, nrm = nr, itm = iters;  // this world's first row in the pool; the warp's rows, rounds and sweeps
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const int o = __shfl_sync(FULL, nact, k * S);
    if (k < sub) base += o;
    rows += o;
  }
#pragma unroll
  for (int o = 16; o >= S; o >>= 1) {
    nrm = max(nrm, __shfl_xor_sync(FULL, nrm, o));
    itm = max(itm, __shfl_xor_sync(FULL, itm, o));
  }
  // the schedule and all rows but FARS in a hundred fit (uniform over the warp;
  // at 25 in a hundred 1000 stacks of 20 took 1046 us an env-step, 987 at 10, at
  // 50 those of 16 1663 in place of 876)
  const bool fits = 100 * (space - ROW_V4 - 16 * nrm) >= (100 - FARS) * ROW_V4 * rows;
  int2* sched = reinterpret_cast<int2*>(zero + ROW_V4) + lane;
  const int head = ROW_V4 + (fits ? 16 * nrm : 0), fit = max(0, min(nact, (space - head) / ROW_V4 - base));
  float4* mine = zero + head + (size_t)base * ROW_V4;
  for (int s = l; s < fit; s += S) {
#pragma unroll
    for (int q = 0; q < ROW_V4; ++q) copy16(mine + (size_t)s * ROW_V4 + q, rec + (size_t)q * nact + s);
  }
  // the lane's part of a round: its row (or none) and that row's body word
  const int* loff = g ? xi + X.scid : nullptr;
  auto row_of = [&](int r) {
    if (r >= nr) return -1;
    const int s = loff[r] + slot;
    return s < loff[r + 1] ? s : -1;
  };
  auto body_of = [&](int word) { return (side ? word >> 8 : word) & 0xff; };
  bool plain = fit == nact && iters == itm;  // every row in the pool, none with pairs that step row by row
  constexpr int STATIC = 1 << 31, FAR = 1 << 30;  // of an accumulator's offset: not written; the row out of line
  if (fits)
    for (int r = 0; r < nrm; ++r) {
      const int s = row_of(r), wd = s < 0 ? 0 : xi[X.ci + s], b = s < 0 ? nb : body_of(wd);
      const bool far = s >= 0 && (s >= fit || wd >= 1 << 16);
      plain = plain && !far;
      sched[32 * r] = make_int2(far ? s : s < 0 ? 0 : (head + (base + s) * ROW_V4) * 16,
                                4 * ACC * b | (b < nb ? 0 : STATIC) | (far ? FAR : 0));
    }
  copies_done();
  __syncwarp();
  auto at_bytes = [](auto* p, int o) { return reinterpret_cast<decltype(p)>(reinterpret_cast<char*>(p) + o); };
  if (fits && __all_sync(FULL, plain)) {
    // The next round's constants are read while this one's update runs, and
    // its offsets a round before that: only the accumulators and the impulses,
    // which the round before may have changed, are waited for.  (Us an
    // env-step without -> with: ten worlds of 16 bodies 104 -> 92, 8192 of 16
    // 577 -> 553, 700 of 53 344 -> 306; at 128 registers, where this spills,
    // 94, 572 and 319.)
    const int2 *at = sched, *end = sched + 32 * nrm;
    auto next = [&]() {
      const int2 c = *at;
      at += 32;
      if (at == end) at = sched;
      return c;
    };
    auto load = [&](int2 c) { return row_load(at_bytes(zero, c.x), 1, side); };
    auto update = [&](const RowRegs& R, int2 c, auto ahead) {
      row_update<false>(R, at_bytes(zero, c.x) + ROW_F4, at_bytes(acc, c.y & ~STATIC), c.y >= 0, 0, side, FULL, ahead);
      __syncwarp();
    };
    int k = itm * nrm;
    if (k > 0) {
      int2 c0 = next(), c1 = next();
      RowRegs R0 = load(c0), R1;
      for (; k > 1; k -= 2) {
        int2 c2;
        update(R0, c0, [&] { R1 = load(c1); c2 = next(); });
        c0 = c2;
        update(R1, c1, [&] { R0 = load(c0); c2 = next(); });
        c1 = c2;
      }
      if (k > 0) update(R0, c0, [] {});
    }
  } else if (fits) {  // the same, then the round's rows that go out of line
    for (int it = 0; it < itm; ++it)
      for (int r = 0; r < nrm; ++r) {
        const int2 c = sched[32 * r];
        const bool on = it < iters, far = on && (c.y & FAR), near = on && !far;
        float4* x = at_bytes(zero, near ? c.x : 0);
        row_update<false>(row_load(x, 1, side), x + ROW_F4, at_bytes(acc, near ? c.y & ~STATIC : 4 * ACC * nbm),
                          near && c.y >= 0, 0, side, FULL, [] {});
        if (__any_sync(FULL, far)) {
          if (far) {
            const bool in = c.x < fit;
            row_update_far(in ? mine + (size_t)c.x * ROW_V4 : rec + c.x, in ? 1 : nact, at_bytes(acc, c.y & ~(STATIC | FAR)),
                           c.y >= 0, xi[X.ci + c.x] >> 16, side, pair);
          }
          __syncwarp();
        }
        __syncwarp();
      }
  } else {
    sweep_mixed(MixedWorld{zero, mine, rec, acc, loff, g ? xi + X.ci : nullptr, fit, nact, nr, iters, nb}, nrm, itm, slot, side);
  }
  if (!g) return;
  const PileLayout& P = g->lay;
  float* F = g->F + (size_t)w * P.fstride;
  int* I = g->I + (size_t)w * P.istride;
  // integration, a lane per body, in the world record
  const float dt = F[P.dtg];
  const V3 grav = v3(F[P.dtg + 1], F[P.dtg + 2], F[P.dtg + 3]);
  const bool rk4 = I[P.integ] == NEWT_INTEGRATOR_RK4;
  bool bad = false;
  for (int b = l; b < nb; b += S) {
    BodyState st{ld3(F + P.pos + 3 * b), ld4(F + P.quat + 4 * b), ld3(F + P.vel + 3 * b), ld3(F + P.omg + 3 * b)};
    const float* u = acc + ACC * b;
    BodyPush f{lds(F + P.inert + 6 * b), lds(F + P.iinv + 6 * b), ld3(u) * sqrtf(1.f / F[P.mass + b]), v3(0.f, 0.f, 0.f)};
    f.dw = qrot(st.q, mv(inverse_inertia_factor(f.iinv), ld3(u + 3)));
    bad |= rk4 ? body_rk4(st, f, dt, grav) : body_euler(st, f, dt, grav);
    st3(F + P.pos + 3 * b, st.p); st3(F + P.vel + 3 * b, st.v); st3(F + P.omg + 3 * b, st.w);
    F[P.quat + 4 * b] = st.q.x; F[P.quat + 4 * b + 1] = st.q.y; F[P.quat + 4 * b + 2] = st.q.z; F[P.quat + 4 * b + 3] = st.q.w;
  }
  if (bad) atomicOr(reinterpret_cast<unsigned*>(I + P.status), NEWT_WS_NONFINITE);
  if (last)
    for (int k = l; k < nact; k += S) {
      const float4 f = k < fit ? mine[(size_t)k * ROW_V4 + ROW_F4] : rec[(size_t)ROW_F4 * nact + k];
      float* o = F + P.imp + P.rpc * xi[X.sccon + k];
      o[0] = f.x; o[1] = f.y; o[2] = f.z; o[3] = f.w;
    }
  if (l == 0) {
    const int con = nact + (first ? 0 : xi[X.misc + B_CON]), rnd = nr + (first ? 0 : xi[X.misc + B_RND]);
    xi[X.misc + B_CON] = con;
    xi[X.misc + B_RND] = rnd;
    if (tally) {
      const unsigned long long rounds = (unsigned long long)rnd * (unsigned long long)max(iters, 0);
      if (cost) cost[flat] = (unsigned)min(rounds + 64ull * (unsigned long long)con, 0xffffffffull);
      atomicAdd(work + 0, (unsigned long long)con);
      if (last) atomicAdd(work + 3, 1ull);
    }
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// The launch shapes the autotuner chooses among: (lanes per world in the
// sweeps, 0 for the class's own; warps per block of pile_k_contacts).
namespace {
struct BatchedShape { int lanes, warps; };
constexpr BatchedShape kShapes[] = {{32, 4}, {16, 4}, {8, 4}, {32, 6}, {16, 8}, {8, 8},
                                    {32, 2}, {16, 2}, {8, 2}, {0, 4},  {0, 8},  {0, 2}};
constexpr int kNumShapes = sizeof(kShapes) / sizeof(kShapes[0]);
constexpr size_t kMostSmem = 227 * 1024 - 1024;
template <class F> void with_sweep(int lanes, F f) {
  if (lanes == 8) f(pile_k_sweep<8>);
  else if (lanes == 16) f(pile_k_sweep<16>);
  else f(pile_k_sweep<32>);
}
}  // namespace

extern "C" int newt_pile_batched_shapes() { return kNumShapes; }

// Size classes of the launches: the largest world of a table sizes every
// world's shared memory.
extern "C" int newt_pile_batched_class(int nb) { return nb <= 8 ? 0 : nb <= 20 ? 1 : 2; }

// The table's launch parameters: lanes per world in the sweeps, warps per
// block and shared words per warp of pile_k_contacts, float4s of rows and
// schedule in the sweeps' shared memory.
struct PileBatchedPlan { int lanes, warps, stride, space, nbm; };

// Shared words per warp of pile_k_contacts for one group's worlds.
extern "C" int newt_pile_batched_words(const PileGroupDev* g) {
  return hot_layout(g->lay, g->nb, g->np, g->maxc).words;
}

// Plans the launches over `worlds` worlds of at most nbm bodies, cm contacts
// and `stride` shared words, and sets the kernels' shared-memory limits (outside stream capture).
// `alone`: no other worlds step beside them.
extern "C" cudaError_t newt_pile_batched_plan(int shape, int worlds, int sms, int nbm, int cm, int stride, bool alone,
                                              PileBatchedPlan* p) {
  const BatchedShape s = kShapes[shape % kNumShapes];
  p->nbm = nbm;
  p->lanes = s.lanes ? s.lanes : nbm > 20 || worlds <= 4 * sms ? 32 : 16;
  p->stride = stride;
  p->warps = s.warps;
  while (p->warps > 1 && (size_t)p->warps * p->stride * 4 > kMostSmem / 2) p->warps /= 2;
  if (worlds <= 4 * sms) p->warps = 1;  // a block each: none waits at another's phase barriers
  // Rows: a settled pile has 1.5 active contacts per body, its worlds spread
  // by 0.4, smaller piles by more; a block of n worlds takes the mean and two
  // and a half deviations (the rest of the space, the other worlds' rounds),
  // three and a half where several worlds share a block and the chip, since a
  // row past the space slows every world of its block.  Rounds: twice the five
  // of 16 bodies, the nine of 53.  Us an env-step at two and a half deviations
  // of 0.4 whatever the size -> now: 3000 worlds of 8 boxes 263 -> 186, 4000 of
  // 12 307 -> 241, 5000 of 14 414 -> 305, 4000 of 16 369 -> 276, 3000 of 18
  // 418 -> 265, 8192 of 16 505 -> 504; beside larger worlds the wider blocks
  // took their place (6000 mixed worlds 364 -> 394).
  const int n = 32 / p->lanes;
  auto space = [&](float spread) {
    const int rows = std::min(n * cm, (int)(nbm * (1.5f * n + spread * sqrtf((float)n))) + 4 + std::max(0, 16 - nbm));
    return ROW_V4 * (rows + 1) + 16 * (10 + nbm / 4) * (n > 2 ? 3 : 2) / 2;
  };
  p->space = space((alone && n > 1 ? 1.4f : 1.f) + 0.2f * std::max(0, 16 - nbm));
  // One world a block: where a deviation less lets the chip hold all blocks at
  // once it is given up (700 worlds of 53 bodies, five an SM in place of four,
  // 289 -> 252 us an env-step).  Two worlds a block lose more by rows past the
  // space (2500 of 16 bodies, nine an SM: 281 -> 311; 8192 of 16 at half a
  // deviation less 507 -> 561).
  if (n == 1) {
    const int per_sm = (worlds + sms - 1) / sms;
    const long all = (227 * 1024 / per_sm - 1024 - (long)sweep_smem(p->lanes, nbm, 0)) / 16;
    if (all >= space(0.6f)) p->space = (int)std::min<long>(p->space, all);
  }
  while (sweep_smem(p->lanes, nbm, p->space) > kMostSmem) p->space /= 2;
  cudaError_t e = cudaFuncSetAttribute(pile_k_contacts, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMostSmem);
  with_sweep(p->lanes, [&](auto kern) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMostSmem);
  });
  return e;
}

// One graph's launches on `st`: the queue sort by its last replay's costs (when
// `cost` and `queue` are given), then two per env-step.  Every live world of
// the table advances `n_steps` env-steps; `end`: the call's last.
extern "C" int newt_launch_pile_batched(const PileGroupDev* dG, const int* dwseg, int ng, int* queue, int n,
                                        int n_steps, int end, unsigned long long* work, unsigned* cost,
                                        const PileBatchedPlan* p, cudaStream_t st) {
  if (n <= 0) return 0;
  int launches = 0;
  if (queue) {
    pile_k_queue_sort<<<1, 1024, 0, st>>>(cost, n, queue);
    ++launches;
  }
  const Worlds W{dG, dwseg, ng, queue, n};
  const int per = 32 / p->lanes;
  for (int s = 0; s < n_steps; ++s) {
    const int tally = s == n_steps - 1, last = tally && end;
    pile_k_contacts<<<(n + p->warps - 1) / p->warps, 32 * p->warps, (size_t)p->warps * p->stride * 4, st>>>(
        W, p->lanes / 2, p->stride, last, work);
    with_sweep(p->lanes, [&](auto kern) {
      kern<<<(n + per - 1) / per, 32, sweep_smem(p->lanes, p->nbm, p->space), st>>>(W, p->nbm, p->space, s == 0, tally, last, work,
                                                                                        cost);
    });
    launches += 2;
  }
  return launches;
}
