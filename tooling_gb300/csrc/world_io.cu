// Per-world I/O, of the named worlds' rows alone (what newt's
// World::apply_mujoco_qpos/qvel, newt/src/world.rs:519-623, touches for one
// world) instead of whole groups.
//
// State and forces are converted on the device from and to the caller's arrays
// (second half of this file).  Models and accelerations move between the host
// mirror and the device: one call packs every group's segment into one pinned
// staging buffer, makes one copy and one scatter (or gather) launch per group,
// then synchronises once; a group whose named worlds are consecutive indices
// skips the packing and moves by one strided copy.  The packed order follows
// the device layout so both sides of each launch are coalesced: tree groups
// keep fields as rows x cap (packed as rows x k), pile groups keep worlds
// contiguous (packed as k x rows).
#include <cuda.h>

#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "host_range.h"
#include "runtime.h"

#define CKW(call)                                                               \
  do {                                                                          \
    cudaError_t e_ = (call);                                                    \
    if (e_ != cudaSuccess) { ctx->err = std::string(#call ": ") + cudaGetErrorString(e_); return NEWT_E_CUDA; } \
  } while (0)

namespace {

__global__ void rows_scatter(float* __restrict__ dF, int soa, int cap, int frows, int lo, int cnt,
                             const int* __restrict__ idx, int k, const float* __restrict__ src) {
  const long total = (long)k * cnt;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x) {
    if (soa) {
      const int r = (int)(t / k), j = (int)(t % k);
      dF[(size_t)(lo + r) * cap + idx[j]] = src[t];
    } else {
      const int j = (int)(t / cnt), r = (int)(t % cnt);
      dF[(size_t)idx[j] * frows + lo + r] = src[t];
    }
  }
}

__global__ void rows_gather(const float* __restrict__ dF, int soa, int cap, int frows, int lo, int cnt,
                            const int* __restrict__ idx, int k, float* __restrict__ dst) {
  const long total = (long)k * cnt;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x) {
    if (soa) {
      const int r = (int)(t / k), j = (int)(t % k);
      dst[t] = dF[(size_t)(lo + r) * cap + idx[j]];
    } else {
      const int j = (int)(t / cnt), r = (int)(t % cnt);
      dst[t] = dF[(size_t)idx[j] * frows + lo + r];
    }
  }
}

__global__ void flags_clear(int* const* __restrict__ flags, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) *flags[i] = 0;
}

int grid_for(long total) {
  const long b = (total + 255) / 256;
  return (int)std::max<long>(1, std::min<long>(b, 152L * 16));
}

// staging: [idx ints | floats], both for every segment of the call; the
// device's half where a call copies into it
int ensure_staging(newt_gpu_ctx* ctx, size_t n_idx, size_t n_f, bool device = true) {
  const size_t bytes = ((n_idx * sizeof(int) + 255) & ~(size_t)255) + n_f * sizeof(float);
  auto grown = [&](size_t held) { return std::max<size_t>(std::max<size_t>(bytes, 2 * held), 1 << 20); };
  if (bytes > ctx->io_bytes) {
    const size_t want = grown(ctx->io_bytes);
    if (ctx->io_h) cudaFreeHost(ctx->io_h);
    ctx->io_h = nullptr;
    ctx->io_bytes = 0;
    CKW(cudaMallocHost(&ctx->io_h, want));
    ctx->io_bytes = want;
  }
  if (device && bytes > ctx->io_d_bytes) {
    const size_t want = grown(ctx->io_d_bytes);
    if (ctx->io_d) cudaFree(ctx->io_d);
    ctx->io_d = nullptr;
    ctx->io_d_bytes = 0;
    CKW(cudaMalloc(&ctx->io_d, want));
    ctx->io_d_bytes = want;
  }
  return NEWT_OK;
}

struct Layout {
  size_t idx_bytes;
  std::vector<size_t> ioff, foff;
  size_t n_idx = 0, n_f = 0;
};

Layout layout(const std::vector<RowMove>& mv) {
  Layout L;
  for (const RowMove& m : mv) {
    L.ioff.push_back(L.n_idx);
    L.foff.push_back(L.n_f);
    L.n_idx += m.idx.size();
    L.n_f += m.idx.size() * m.cnt;
  }
  L.idx_bytes = (L.n_idx * sizeof(int) + 255) & ~(size_t)255;
  return L;
}

// A world list that is one run of consecutive indices moves as one strided
// copy straight between the host mirror and the device, with no packing.
bool consecutive(const std::vector<int>& idx) {
  for (size_t j = 1; j < idx.size(); ++j)
    if (idx[j] != idx[0] + (int)j) return false;
  return !idx.empty();
}

cudaError_t copy_run(const RowMove& m, cudaStream_t st, bool to_device) {
  HostGroup& g = *m.g;
  const size_t a = (size_t)m.idx[0], k = m.idx.size();
  float* h = m.ints ? reinterpret_cast<float*>(g.hI.data()) : g.hF.data();
  float* d = m.ints ? reinterpret_cast<float*>(g.dI) : g.dF;
  const size_t rows = m.ints ? g.irows : g.frows;
  if (g.soa()) {  // cnt rows of k consecutive worlds, row pitch cap
    const size_t off = m.lo * g.cap + a, pitch = g.cap * sizeof(float);
    return to_device ? cudaMemcpy2DAsync(d + off, pitch, h + off, pitch, k * sizeof(float), m.cnt,
                                         cudaMemcpyHostToDevice, st)
                     : cudaMemcpy2DAsync(h + off, pitch, d + off, pitch, k * sizeof(float), m.cnt,
                                         cudaMemcpyDeviceToHost, st);
  }
  const size_t off = a * rows + m.lo, pitch = rows * sizeof(float);  // k worlds of cnt values
  return to_device ? cudaMemcpy2DAsync(d + off, pitch, h + off, pitch, m.cnt * sizeof(float), k,
                                       cudaMemcpyHostToDevice, st)
                   : cudaMemcpy2DAsync(h + off, pitch, d + off, pitch, m.cnt * sizeof(float), k,
                                       cudaMemcpyDeviceToHost, st);
}

}  // namespace

int io_scatter(newt_gpu_ctx* ctx, const std::vector<RowMove>& all) {
  std::vector<RowMove> mv;
  for (const RowMove& m : all) {
    if (consecutive(m.idx)) CKW(copy_run(m, ctx->stream, true));
    else mv.push_back(m);
  }
  if (mv.empty()) {
    CKW(cudaStreamSynchronize(ctx->stream));
    return NEWT_OK;
  }
  const Layout L = layout(mv);
  int rc = ensure_staging(ctx, L.n_idx, L.n_f);
  if (rc != NEWT_OK) return rc;
  int* hi = (int*)ctx->io_h;
  float* hf = (float*)((char*)ctx->io_h + L.idx_bytes);
  for (size_t s = 0; s < mv.size(); ++s) {
    const RowMove& m = mv[s];
    const HostGroup& g = *m.g;
    const size_t k = m.idx.size();
    std::copy(m.idx.begin(), m.idx.end(), hi + L.ioff[s]);
    float* out = hf + L.foff[s];
    for (size_t j = 0; j < k; ++j)
      for (size_t r = 0; r < m.cnt; ++r) {
        float v;
        if (m.ints) { const int iv = g.Ic(m.lo + r, m.idx[j]); std::memcpy(&v, &iv, sizeof(v)); }
        else v = g.Fc(m.lo + r, m.idx[j]);
        if (g.soa()) out[r * k + j] = v; else out[j * m.cnt + r] = v;
      }
  }
  CKW(cudaMemcpyAsync(ctx->io_d, ctx->io_h, L.idx_bytes + L.n_f * sizeof(float), cudaMemcpyHostToDevice, ctx->stream));
  const int* di = (const int*)ctx->io_d;
  const float* df = (const float*)((char*)ctx->io_d + L.idx_bytes);
  for (size_t s = 0; s < mv.size(); ++s) {
    const RowMove& m = mv[s];
    const long total = (long)m.idx.size() * m.cnt;
    if (total == 0) continue;
    rows_scatter<<<grid_for(total), 256, 0, ctx->stream>>>(m.ints ? reinterpret_cast<float*>(m.g->dI) : m.g->dF,
                                                            m.g->soa() ? 1 : 0, m.g->cap,
                                                            (int)(m.ints ? m.g->irows : m.g->frows),
                                                            (int)m.lo, (int)m.cnt, di + L.ioff[s], (int)m.idx.size(),
                                                            df + L.foff[s]);
    ctx->launches++;
  }
  CKW(cudaGetLastError());
  CKW(cudaStreamSynchronize(ctx->stream));  // the pinned staging is reused by the next call
  return NEWT_OK;
}

int io_gather(newt_gpu_ctx* ctx, const std::vector<RowMove>& all) {
  std::vector<RowMove> mv;
  for (const RowMove& m : all) {
    if (consecutive(m.idx)) CKW(copy_run(m, ctx->stream, false));
    else mv.push_back(m);
  }
  if (mv.empty()) {
    CKW(cudaStreamSynchronize(ctx->stream));
    return NEWT_OK;
  }
  const Layout L = layout(mv);
  int rc = ensure_staging(ctx, L.n_idx, L.n_f);
  if (rc != NEWT_OK) return rc;
  int* hi = (int*)ctx->io_h;
  for (size_t s = 0; s < mv.size(); ++s) std::copy(mv[s].idx.begin(), mv[s].idx.end(), hi + L.ioff[s]);
  CKW(cudaMemcpyAsync(ctx->io_d, ctx->io_h, L.n_idx * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
  const int* di = (const int*)ctx->io_d;
  float* df = (float*)((char*)ctx->io_d + L.idx_bytes);
  for (size_t s = 0; s < mv.size(); ++s) {
    const RowMove& m = mv[s];
    const long total = (long)m.idx.size() * m.cnt;
    if (total == 0) continue;
    rows_gather<<<grid_for(total), 256, 0, ctx->stream>>>(m.ints ? reinterpret_cast<const float*>(m.g->dI) : m.g->dF,
                                                           m.g->soa() ? 1 : 0, m.g->cap,
                                                           (int)(m.ints ? m.g->irows : m.g->frows),
                                                           (int)m.lo, (int)m.cnt, di + L.ioff[s], (int)m.idx.size(),
                                                           df + L.foff[s]);
    ctx->launches++;
  }
  CKW(cudaGetLastError());
  float* hf = (float*)((char*)ctx->io_h + L.idx_bytes);
  CKW(cudaMemcpyAsync(hf, df, L.n_f * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
  CKW(cudaStreamSynchronize(ctx->stream));
  for (size_t s = 0; s < mv.size(); ++s) {
    const RowMove& m = mv[s];
    HostGroup& g = *m.g;
    const size_t k = m.idx.size();
    const float* in = hf + L.foff[s];
    for (size_t j = 0; j < k; ++j)
      for (size_t r = 0; r < m.cnt; ++r) {
        const float v = g.soa() ? in[r * k + j] : in[j * m.cnt + r];
        if (m.ints) std::memcpy(&g.I(m.lo + r, m.idx[j]), &v, sizeof(v));
        else g.F(m.lo + r, m.idx[j]) = v;
      }
  }
  return NEWT_OK;
}

// ---------------------------------------------------------------------------
// state and forces in MuJoCo layout, converted on the device
// ---------------------------------------------------------------------------
// newt_gpu_set_state / get_state / set_qfrc convert between the caller's
// MuJoCo-layout arrays and the groups' rows in one launch: quaternions
// reordered (wxyz <-> xyzw) and, on the way in, normalised; a free root's
// linear velocity rotated between world and body frame (newt's
// apply_mujoco_qpos/qvel, world.rs:519-623, and its inverse).  A free root's
// and a hinge's MuJoCo offsets equal newt's (7 and 1 coordinates, 6 and 1
// rates), so a link's `topo` offsets index both layouts.
//
// What bounds a call: latency for few worlds (the launch, the wait), the host's loops over the slots and the link
// for many.  So
//   * the worlds are taken as runs of consecutive indices in a group, a few
//     of which describe most calls and travel as kernel parameters (up to
//     128; a table in the staging past that); worlds named in no order, fewer
//     than eight a run, go by a list in the staging instead, a warp each (runs
//     cost a block and 120 bytes apiece: 16384 quadrupeds shuffled, set_state
//     444 us as runs of one and 189 by the list, 152 and 119 as runs of four,
//     118 and 115 as runs of eight; 512 chains, runs of eight 24 and 24);
//   * a call for forces skips free bodies, which carry none;
//   * page-locked arrays are read and written by the kernel itself, others
//     through the page-locked staging;
//   * a block moves up to 32 worlds of a run by way of shared memory, so that
//     both the caller's array (worlds one after another) and a tree group's
//     rows (worlds side by side) are touched in whole lines.
// Measured (GB300, us for set_state and get_state from page-locked arrays; one
// plan entry per world and a copy per array before -> now): 16384 quadrupeds
// 212 and 206 -> 81 and 81 (set_qfrc from an ordinary array, which went by way
// of a host transpose, 423 -> 127), 8192 piles of 16 153 and 153 -> 81 and 81,
// 6000 mixed worlds 128 and 130 -> 63 and 61, one pendulum 24 and 22 -> 19 and
// 18.
namespace {

struct StateRun {
  float* F;
  const int* topo;                // tree: parent, joint, q offset, v offset per link
  long frows, q0, v0;             // the run's first coordinate and rate in the caller's arrays
  int soa, cap, size, nq, nv;     // tree SoA (row * cap + w) or pile world-major (w * frows + row); bodies or links
  int pos, quat, vel, omg;        // pile rows
  int rq, rqd, rf;                // tree rows: coordinates, rates, applied forces
  int w0, n, tile, blk;           // first index, worlds, worlds per block, first block
};
template <int N>
struct StateRuns { int n; StateRun r[N]; };
enum StateMove { STATE_IN, STATE_OUT, QFRC_IN };
constexpr int TILE_FLOATS = 10240;  // a block's share of the arrays (40 KB of shared memory)

NEWT_D float& frow(const StateRun& g, int row, int w) {
  return g.soa ? g.F[(size_t)row * g.cap + w] : g.F[(size_t)w * g.frows + row];
}
NEWT_D Q4 qnorm_or_identity(Q4 q) {  // the host's q_norm: a zero quaternion becomes the identity
  const float n = sqrtf(q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w);
  return n == 0.f ? Q4{0.f, 0.f, 0.f, 1.f} : Q4{q.x / n, q.y / n, q.z / n, q.w / n};
}

// Body or link i of world w: its coordinates at qp and rates at qv to the rows.
NEWT_D void state_in(const StateRun& g, int i, int w, const float* qp, const float* qv) {
  if (!g.soa) {  // free body i
    const float* p = qp + 7 * i;
    const float* v = qv + 6 * i;
    const Q4 q = qnorm_or_identity(Q4{p[4], p[5], p[6], p[3]});
    for (int k = 0; k < 3; ++k) {
      frow(g, g.pos + 3 * i + k, w) = p[k];
      frow(g, g.vel + 3 * i + k, w) = v[k];
      frow(g, g.omg + 3 * i + k, w) = v[3 + k];
    }
    frow(g, g.quat + 4 * i, w) = q.x; frow(g, g.quat + 4 * i + 1, w) = q.y;
    frow(g, g.quat + 4 * i + 2, w) = q.z; frow(g, g.quat + 4 * i + 3, w) = q.w;
    return;
  }
  const int jt = g.topo[4 * i + 1], qo = g.topo[4 * i + 2], vo = g.topo[4 * i + 3];
  if (jt == NEWT_JOINT_FREE) {  // pos, quat xyzw; omega_body, v_body
    const Q4 q = qnorm_or_identity(Q4{qp[qo + 4], qp[qo + 5], qp[qo + 6], qp[qo + 3]});
    const V3 vb = qrot_inv(q, v3(qv[vo], qv[vo + 1], qv[vo + 2]));
    for (int k = 0; k < 3; ++k) frow(g, g.rq + qo + k, w) = qp[qo + k];
    frow(g, g.rq + qo + 3, w) = q.x; frow(g, g.rq + qo + 4, w) = q.y;
    frow(g, g.rq + qo + 5, w) = q.z; frow(g, g.rq + qo + 6, w) = q.w;
    for (int k = 0; k < 3; ++k) frow(g, g.rqd + vo + k, w) = qv[vo + 3 + k];
    frow(g, g.rqd + vo + 3, w) = vb.x; frow(g, g.rqd + vo + 4, w) = vb.y; frow(g, g.rqd + vo + 5, w) = vb.z;
  } else if (jt == NEWT_JOINT_HINGE || jt == NEWT_JOINT_SLIDE) {
    frow(g, g.rq + qo, w) = qp[qo];
    frow(g, g.rqd + vo, w) = qv[vo];
  }
}
NEWT_D void state_out(const StateRun& g, int i, int w, float* qp, float* qv) {
  if (!g.soa) {
    float* p = qp + 7 * i;
    float* v = qv + 6 * i;
    for (int k = 0; k < 3; ++k) {
      p[k] = frow(g, g.pos + 3 * i + k, w);
      v[k] = frow(g, g.vel + 3 * i + k, w);
      v[3 + k] = frow(g, g.omg + 3 * i + k, w);
    }
    p[3] = frow(g, g.quat + 4 * i + 3, w); p[4] = frow(g, g.quat + 4 * i, w);
    p[5] = frow(g, g.quat + 4 * i + 1, w); p[6] = frow(g, g.quat + 4 * i + 2, w);
    return;
  }
  const int jt = g.topo[4 * i + 1], qo = g.topo[4 * i + 2], vo = g.topo[4 * i + 3];
  if (jt == NEWT_JOINT_FREE) {
    const Q4 q{frow(g, g.rq + qo + 3, w), frow(g, g.rq + qo + 4, w), frow(g, g.rq + qo + 5, w),
               frow(g, g.rq + qo + 6, w)};
    for (int k = 0; k < 3; ++k) qp[qo + k] = frow(g, g.rq + qo + k, w);
    qp[qo + 3] = q.w; qp[qo + 4] = q.x; qp[qo + 5] = q.y; qp[qo + 6] = q.z;
    const V3 vw = qrot(q, v3(frow(g, g.rqd + vo + 3, w), frow(g, g.rqd + vo + 4, w), frow(g, g.rqd + vo + 5, w)));
    qv[vo] = vw.x; qv[vo + 1] = vw.y; qv[vo + 2] = vw.z;
    for (int k = 0; k < 3; ++k) qv[vo + 3 + k] = frow(g, g.rqd + vo + k, w);
  } else if (jt == NEWT_JOINT_HINGE || jt == NEWT_JOINT_SLIDE) {
    qp[qo] = frow(g, g.rq + qo, w);
    qv[vo] = frow(g, g.rqd + vo, w);
  }
}

template <int MOVE>
NEWT_D void move_tile(const StateRun* runs, int n, float* qpos, float* qvel) {
  extern __shared__ float tile_s[];
  int lo = 0, hi = n - 1;  // the run this block's first block count falls in
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (runs[mid].blk <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const StateRun g = runs[lo];
  const int base = ((int)blockIdx.x - g.blk) * g.tile, T = min(g.tile, g.n - base), w0 = g.w0 + base;
  const int nq = MOVE == QFRC_IN ? 0 : g.nq, nv = g.nv, tid = threadIdx.x, nt = blockDim.x;
  float* sq = tile_s;
  float* sv = tile_s + g.tile * nq;
  float* q = qpos + g.q0 + (long)base * nq;
  float* v = qvel + g.v0 + (long)base * nv;
  if (MOVE != STATE_OUT) {
    for (int e = tid; e < T * nq; e += nt) sq[e] = q[e];
    for (int e = tid; e < T * nv; e += nt) sv[e] = v[e];
    __syncthreads();
  }
  if (MOVE == QFRC_IN) {
    for (int e = tid; e < 32 * nv; e += nt)  // of trees alone
      if ((e & 31) < T) frow(g, g.rf + (e >> 5), w0 + (e & 31)) = sv[(e & 31) * nv + (e >> 5)];
    return;
  }
  if (g.soa) {  // worlds side by side (a tile of at most 32)
    for (int e = tid; e < 32 * g.size; e += nt) {
      const int j = e & 31, i = e >> 5;
      if (j >= T) continue;
      if (MOVE == STATE_IN) state_in(g, i, w0 + j, sq + j * nq, sv + j * nv);
      else state_out(g, i, w0 + j, sq + j * nq, sv + j * nv);
    }
  } else {
    for (int e = tid; e < T * g.size; e += nt) {
      const int j = e / g.size, i = e % g.size;
      if (MOVE == STATE_IN) state_in(g, i, w0 + j, sq + j * nq, sv + j * nv);
      else state_out(g, i, w0 + j, sq + j * nq, sv + j * nv);
    }
  }
  if (MOVE == STATE_OUT) {
    __syncthreads();
    for (int e = tid; e < T * nq; e += nt) q[e] = sq[e];
    for (int e = tid; e < T * nv; e += nt) v[e] = sv[e];
  }
}
// A world of a call that names them in no order: its group's entry, its index,
// its first coordinate and rate in the caller's arrays.
struct StateWorld { int g, w; long q0, v0; };
constexpr int LIST_WARPS = 8, LIST_RUN = 8;
// A warp per listed world, by way of `per` floats of shared memory each.
template <int MOVE>
__global__ void __launch_bounds__(32 * LIST_WARPS) state_move_list(const StateRun* G, const StateWorld* W, int n, int per,
                                                                   float* qpos, float* qvel) {
  extern __shared__ float tile_s[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = blockIdx.x * LIST_WARPS + warp;
  if (t >= n) return;
  const StateWorld sw = W[t];
  const StateRun& g = G[sw.g];
  const int nq = g.nq, nv = g.nv, w = sw.w;
  float* q = qpos + sw.q0;
  float* v = qvel + sw.v0;
  if (MOVE == QFRC_IN) {
    for (int k = lane; k < nv; k += 32) frow(g, g.rf + k, w) = v[k];
    return;
  }
  float* sq = tile_s + warp * per;
  float* sv = sq + nq;
  if (MOVE == STATE_IN) {
    for (int k = lane; k < nq; k += 32) sq[k] = q[k];
    for (int k = lane; k < nv; k += 32) sv[k] = v[k];
    __syncwarp();
    for (int i = lane; i < g.size; i += 32) state_in(g, i, w, sq, sv);
  } else {
    for (int i = lane; i < g.size; i += 32) state_out(g, i, w, sq, sv);
    __syncwarp();
    for (int k = lane; k < nq; k += 32) q[k] = sq[k];
    for (int k = lane; k < nv; k += 32) v[k] = sv[k];
  }
}
template <int MOVE, int N>
__global__ void __launch_bounds__(256) state_move(const __grid_constant__ StateRuns<N> R, float* qpos, float* qvel) {
  move_tile<MOVE>(R.r, R.n, qpos, qvel);
}
template <int MOVE>
__global__ void __launch_bounds__(256) state_move_table(const StateRun* R, int n, float* qpos, float* qvel) {
  move_tile<MOVE>(R, n, qpos, qvel);
}

// The device's address of n floats of page-locked host memory, or null: the
// kernels read and write the caller's array in place only where one
// page-locked range holds all of it.
HostRange host_range(const void* p) {
  using Get = CUresult (*)(unsigned, CUpointer_attribute*, void**, CUdeviceptr);
  static const Get get = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &f, 12000, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      f = nullptr;
    }
    return reinterpret_cast<Get>(f);
  }();
  cudaPointerAttributes a;
  if (!get || cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return HostRange{};
  }
  if (a.type != cudaMemoryTypeHost || !a.devicePointer) return HostRange{};
  CUdeviceptr start = 0;
  size_t bytes = 0;
  CUpointer_attribute what[2] = {CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE};
  void* out[2] = {&start, &bytes};
  if (get(2, what, out, (CUdeviceptr)a.devicePointer) != CUDA_SUCCESS) return HostRange{};
  return HostRange{(uintptr_t)a.devicePointer, (uintptr_t)start, bytes};
}
float* device_view(const void* p, size_t n) {
  if (n == 0 || ((uintptr_t)p & 3)) return nullptr;
  return reinterpret_cast<float*>(device_address(p, n * sizeof(float), host_range));
}

size_t up256(size_t b) { return (b + 255) & ~(size_t)255; }

// The call's worlds as runs of consecutive indices in a group.  Slots are
// named in ascending order when none can be named twice.
struct Run { int group, w0, n, nq, nv; long q0, v0; };
struct StatePlan {
  std::vector<Run> runs;
  long nq = 0, nv = 0;
  int worlds = 0;
  bool ascending = true;
  // Worlds in no order (a run for every few of them) move by a list, a warp
  // each; see state_move_list.
  bool listed() const { return runs.size() > 128 && runs.size() * LIST_RUN > (size_t)worlds; }
};
// `forces`: only the worlds that carry generalised forces.  `skip` (nullable):
// a flag per named slot, those to pass over.
int plan_state(newt_gpu_ctx* ctx, const int32_t* slots, int n, bool forces, const char* skip, StatePlan& P) {
  const int n_slots = (int)ctx->slots.size();
  const SlotRef* refs = ctx->slots.data();
  int group = -1, next = -1, prev = -1, nq = 0, nv = 0;
  bool moves = true, open = false;  // the group's worlds move; the last run takes its next one
  Run run{};
  for (int i = 0; i < n; ++i) {
    const int s = slots[i];
    if (s < 0 || s >= n_slots || !refs[s].live) {
      ctx->err = "bad slot";
      return NEWT_E_INVALID;
    }
    P.ascending = P.ascending && s > prev;
    prev = s;
    if (refs[s].group != group) {
      group = refs[s].group;
      const HostGroup& hg = *ctx->groups[group];
      nq = hg.nq;
      nv = hg.nv;
      moves = !forces || hg.soa();
      next = -1;
    }
    if (!moves || (skip && skip[i])) {
      next = -1;
    } else {
      if (refs[s].index != next) {
        if (open) {
          if (P.runs.size() == 128) P.runs.reserve(n);  // they keep coming
          P.runs.push_back(run);
        }
        open = true;
        run = Run{group, refs[s].index, 0, nq, nv, P.nq, P.nv};
        next = run.w0;
      }
      ++run.n;
      ++next;
      ++P.worlds;
    }
    P.nq += nq;
    P.nv += nv;
  }
  if (open) P.runs.push_back(run);
  return NEWT_OK;
}

// What the kernels take of a run.
StateRun describe(newt_gpu_ctx* ctx, const Run& r) {
  const HostGroup& hg = *ctx->groups[r.group];
  StateRun g{};
  g.F = hg.dF;
  g.topo = hg.dtopo;
  g.frows = (long)hg.frows;
  g.soa = hg.soa() ? 1 : 0;
  g.cap = hg.cap;
  g.size = hg.size;
  g.nq = r.nq;
  g.nv = r.nv;
  g.q0 = r.q0;
  g.v0 = r.v0;
  g.w0 = r.w0;
  g.n = r.n;
  g.pos = hg.lay.pos; g.quat = hg.lay.quat; g.vel = hg.lay.vel; g.omg = hg.lay.omg;
  g.rq = hg.r_q; g.rqd = hg.r_qd; g.rf = hg.r_qfrc;
  return g;
}

template <int MOVE, int N>
void launch_runs(const StateRun* runs, int n, int blocks, size_t smem, float* q, float* v, cudaStream_t st) {
  StateRuns<N> R;
  R.n = n;
  std::copy(runs, runs + n, R.r);
  state_move<MOVE, N><<<blocks, 256, smem, st>>>(R, q, v);
}

// Bytes of the staging's head (host and device) that the move takes.
size_t table_bytes(newt_gpu_ctx* ctx, const StatePlan& P) {
  if (P.listed()) return up256(ctx->groups.size() * sizeof(StateRun)) + up256(P.worlds * sizeof(StateWorld));
  return P.runs.size() > 128 ? up256(P.runs.size() * sizeof(StateRun)) : 0;
}

// Moves the planned worlds between the rows and the arrays at device
// addresses q and v.
template <int MOVE>
int move_worlds(newt_gpu_ctx* ctx, const StatePlan& P, float* q, float* v) {
  if (P.worlds == 0) return NEWT_OK;
  char* h = (char*)ctx->io_h;
  char* d = (char*)ctx->io_d;
  if (P.listed()) {
    const size_t head = up256(ctx->groups.size() * sizeof(StateRun));
    StateRun* hg = (StateRun*)h;
    StateWorld* hw = (StateWorld*)(h + head);
    std::vector<int> entry(ctx->groups.size(), -1);
    int groups = 0, per = 1;
    for (const Run& r : P.runs) {
      if (entry[r.group] < 0) {
        hg[groups] = describe(ctx, r);
        per = std::max(per, r.nq + r.nv);
        entry[r.group] = groups++;
      }
      for (int k = 0; k < r.n; ++k) *hw++ = StateWorld{entry[r.group], r.w0 + k, r.q0 + (long)k * r.nq, r.v0 + (long)k * r.nv};
    }
    CKW(cudaMemcpyAsync(d, h, groups * sizeof(StateRun), cudaMemcpyHostToDevice, ctx->stream));
    // the list is read once, where it lies
    const StateWorld* dw = (const StateWorld*)device_view(h + head, P.worlds * sizeof(StateWorld) / sizeof(float));
    state_move_list<MOVE><<<(P.worlds + LIST_WARPS - 1) / LIST_WARPS, 32 * LIST_WARPS,
                            MOVE == QFRC_IN ? 0 : LIST_WARPS * per * sizeof(float), ctx->stream>>>(
        (const StateRun*)d, dw, P.worlds, per, q, v);
  } else {
    std::vector<StateRun> runs;
    runs.reserve(P.runs.size());
    int blocks = 0;
    size_t smem = 0;
    for (const Run& r : P.runs) {
      StateRun g = describe(ctx, r);
      const int per = std::max(1, (MOVE == QFRC_IN ? 0 : g.nq) + g.nv);
      g.tile = std::min(32, std::max(1, TILE_FLOATS / per));
      g.blk = blocks;
      blocks += (g.n + g.tile - 1) / g.tile;
      smem = std::max(smem, (size_t)g.tile * per * sizeof(float));
      runs.push_back(g);
    }
    const int n = (int)runs.size();
    if (n <= 2) {
      launch_runs<MOVE, 2>(runs.data(), n, blocks, smem, q, v, ctx->stream);
    } else if (n <= 24) {
      launch_runs<MOVE, 24>(runs.data(), n, blocks, smem, q, v, ctx->stream);
    } else if (n <= 128) {
      launch_runs<MOVE, 128>(runs.data(), n, blocks, smem, q, v, ctx->stream);
    } else {
      std::copy(runs.begin(), runs.end(), (StateRun*)h);
      CKW(cudaMemcpyAsync(d, h, n * sizeof(StateRun), cudaMemcpyHostToDevice, ctx->stream));
      state_move_table<MOVE><<<blocks, 256, smem, ctx->stream>>>((const StateRun*)d, n, q, v);
    }
  }
  ctx->launches++;
  CKW(cudaGetLastError());
  return NEWT_OK;
}

// A slot named twice?
bool repeats(newt_gpu_ctx* ctx, const int32_t* slots, int n) {
  std::vector<char> seen(ctx->slots.size(), 0);
  for (int i = 0; i < n; ++i) {
    if (seen[slots[i]]) return true;
    seen[slots[i]] = 1;
  }
  return false;
}

// The arrays as the device reaches them: page-locked ones as they are, others
// by the staging, past the run table.
struct Views { float *q = nullptr, *v = nullptr; bool q_staged = false, v_staged = false; size_t qo = 0, vo = 0; };
int view_arrays(newt_gpu_ctx* ctx, const StatePlan& P, const void* qpos, const void* qvel, Views& w) {
  const size_t table = table_bytes(ctx, P);
  const size_t nq = qpos ? (size_t)P.nq : 0, nv = (size_t)P.nv;
  w.q = device_view(qpos, nq);
  w.v = device_view(qvel, nv);
  w.q_staged = nq > 0 && !w.q;
  w.v_staged = nv > 0 && !w.v;
  w.qo = table;
  w.vo = table + (w.q_staged ? up256(nq * sizeof(float)) : 0);
  const size_t bytes = w.vo + (w.v_staged ? nv * sizeof(float) : 0);
  if (bytes > 0) {
    const int rc = ensure_staging(ctx, 0, bytes / sizeof(float) + 1, table > 0);
    if (rc != NEWT_OK) return rc;
  }
  if (w.q_staged) w.q = device_view((char*)ctx->io_h + w.qo, nq);
  if (w.v_staged) w.v = device_view((char*)ctx->io_h + w.vo, nv);
  return NEWT_OK;
}

}  // namespace

int io_state_in(newt_gpu_ctx* ctx, const int32_t* slots, int n, const float* qpos, const float* qvel) {
  StatePlan P;
  int rc = plan_state(ctx, slots, n, false, nullptr, P);
  if (rc != NEWT_OK) return rc;
  if (!P.ascending && repeats(ctx, slots, n)) {
    ctx->err = "slot named twice";
    return NEWT_E_INVALID;
  }
  Views w;
  if ((rc = view_arrays(ctx, P, qpos, qvel, w)) != NEWT_OK) return rc;
  if (w.q_staged) std::memcpy((char*)ctx->io_h + w.qo, qpos, P.nq * sizeof(float));
  if (w.v_staged) std::memcpy((char*)ctx->io_h + w.vo, qvel, P.nv * sizeof(float));
  if ((rc = move_worlds<STATE_IN>(ctx, P, w.q, w.v)) != NEWT_OK) return rc;
  CKW(cudaStreamSynchronize(ctx->stream));  // the caller's arrays and the staging are free again
  return NEWT_OK;
}

int io_state_out(newt_gpu_ctx* ctx, const int32_t* slots, int n, float* qpos, float* qvel) {
  StatePlan P;
  int rc = plan_state(ctx, slots, n, false, nullptr, P);
  if (rc != NEWT_OK) return rc;
  Views w;
  if ((rc = view_arrays(ctx, P, qpos, qvel, w)) != NEWT_OK) return rc;
  if ((rc = move_worlds<STATE_OUT>(ctx, P, w.q, w.v)) != NEWT_OK) return rc;
  CKW(cudaStreamSynchronize(ctx->stream));
  if (w.q_staged) std::memcpy(qpos, (char*)ctx->io_h + w.qo, P.nq * sizeof(float));
  if (w.v_staged) std::memcpy(qvel, (char*)ctx->io_h + w.vo, P.nv * sizeof(float));
  return NEWT_OK;
}

int io_qfrc_in(newt_gpu_ctx* ctx, const int32_t* slots, int n, const float* qfrc) {
  StatePlan P;
  int rc = plan_state(ctx, slots, n, true, nullptr, P);
  if (rc != NEWT_OK) return rc;
  if (!P.ascending && repeats(ctx, slots, n)) {  // a slot named twice keeps the last forces
    std::vector<char> seen(ctx->slots.size(), 0), skip(n, 0);
    for (int i = n - 1; i >= 0; --i) {
      skip[i] = seen[slots[i]];
      seen[slots[i]] = 1;
    }
    P = StatePlan{};
    if ((rc = plan_state(ctx, slots, n, true, skip.data(), P)) != NEWT_OK) return rc;
  }
  if (P.worlds > 0) {  // free bodies alone carry no generalised force
    Views w;
    if ((rc = view_arrays(ctx, P, nullptr, qfrc, w)) != NEWT_OK) return rc;
    if (w.v_staged) {
      float* h = (float*)((char*)ctx->io_h + w.vo);
      for (size_t k = 0; k < P.runs.size();) {  // what is moved, in runs that follow one another
        const long a = P.runs[k].v0;
        long b = a;
        for (; k < P.runs.size() && P.runs[k].v0 == b; ++k) b += (long)P.runs[k].n * P.runs[k].nv;
        std::memcpy(h + a, qfrc + a, (size_t)(b - a) * sizeof(float));
      }
    }
    if ((rc = move_worlds<QFRC_IN>(ctx, P, nullptr, w.v)) != NEWT_OK) return rc;
  }
  CKW(cudaStreamSynchronize(ctx->stream));
  return NEWT_OK;
}

// Up to 1024 live flags cleared by one launch with the pointers passed by
// value (8 KB of parameters): nothing to stage, so the call returns at once.
struct HoldList {
  int n;
  int* f[1024];
};
__global__ void flags_hold(HoldList L) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < L.n) *L.f[i] = 0;
}

int io_hold_flags(newt_gpu_ctx* ctx, const std::vector<int*>& flags) {
  for (size_t a = 0; a < flags.size(); a += 1024) {
    HoldList L;
    L.n = (int)std::min<size_t>(1024, flags.size() - a);
    for (int i = 0; i < L.n; ++i) L.f[i] = flags[a + i];
    flags_hold<<<(L.n + 255) / 256, 256, 0, ctx->stream>>>(L);
    ctx->launches++;
    CKW(cudaGetLastError());
  }
  return NEWT_OK;
}

int io_clear_flags(newt_gpu_ctx* ctx, const std::vector<int*>& flags) {
  if (flags.empty()) return NEWT_OK;
  int rc = ensure_staging(ctx, 0, 2 * flags.size());  // one pointer = two floats' room
  if (rc != NEWT_OK) return rc;
  std::copy(flags.begin(), flags.end(), (int**)ctx->io_h);
  CKW(cudaMemcpyAsync(ctx->io_d, ctx->io_h, flags.size() * sizeof(int*), cudaMemcpyHostToDevice, ctx->stream));
  flags_clear<<<grid_for((long)flags.size()), 256, 0, ctx->stream>>>((int* const*)ctx->io_d, (int)flags.size());
  ctx->launches++;
  CKW(cudaGetLastError());
  CKW(cudaStreamSynchronize(ctx->stream));
  return NEWT_OK;
}
