// hmf_cell.cuh -- the two kernels of an iteration on small volumes, whose
// state stays in L2 and whose cost is latency: launch, copy set-up and the
// serial steps of a z-march.
//
//  flow_cell_kernel  the flow step (flow_tma_kernel's arithmetic, operation by
//                    operation) of one vertex on one 16 x 8 x 4 cell.  A cell's
//                    planes are all formed side by side: four stages over the
//                    cell and its halo -- g, p', m, then P, the divergence and
//                    the stores -- with three CTA barriers in all, where the
//                    march takes one per plane after filling its copy rings.
//                    The halo is recomputed (1920 values of g for 512 outputs),
//                    which pays only while the GPU would be idle.
//  sweep_cell_kernel the sweep (tree_kernel's arithmetic) with one voxel per
//                    thread, every value loaded before the first is used.
//
// Both let the next kernel of the stream start while they run (programmatic
// dependent launch) and wait for the previous one before they touch its
// results, so launch and set-up overlap.
#pragma once

#include "hmf_flow_tma.cuh"
#include "hmf_types.cuh"

namespace hmf {

constexpr int kCellX = 16, kCellY = 8, kCellZ = 4;
constexpr int kCellThreads = 256;

// Staged boxes of a cell: origin `lo` cells below the cell's, extent T + lo + hi.
template <int LO, int HI>
struct CellBox {
  static constexpr int X = kCellX + LO + HI, Y = kCellY + LO + HI, Z = kCellZ + LO + HI;
  static constexpr int N = X * Y * Z;
  static constexpr int SY = X, SZ = X * Y;
  __device__ static int at(int x, int y, int z) { return (x + LO) + (y + LO) * SY + (z + LO) * SZ; }
};

__global__ void __launch_bounds__(kCellThreads)
    flow_cell_kernel(const FlowVertex* __restrict__ vertices, const Geometry G, const FlowParams fp) {
  using BG = CellBox<2, 2>;  // g and p'
  using BM = CellBox<1, 1>;  // m
  __shared__ float g[BG::N], p[3][BG::N], m[BM::N];
  dependents_may_launch();
  const int tiles_y = (G.vy + kCellY - 1) / kCellY;
  const int tx = blockIdx.x % fp.tiles_x, tyz = blockIdx.x / fp.tiles_x;
  const int x0 = tx * kCellX, y0 = (tyz % tiles_y) * kCellY, z0 = (tyz / tiles_y) * kCellZ;
  const float step = fp.step, icc = fp.icc;
  const int plane = (int)G.plane, pitch = G.pitch;
  wait_for_previous_grid();
  // (after the wait: a solve's first launch follows the table's copy)
  const FlowVertex V = vertices[blockIdx.y];
  auto inside = [&](int x, int y, int z) { return x >= 0 && x < G.vx && y >= 0 && y < G.vy && z >= 0 && z < G.vz; };

  // g = step * (((sink + div) - inc) - label * icc), div recomputed from the
  // stored flows as kern_Divergence formed it; the flows are kept.  Loads are
  // clamped into the volume instead of predicated, so that a thread's four
  // points have their 36 loads in flight together.
#pragma unroll 1
  for (int i0 = threadIdx.x; i0 < BG::N; i0 += 4 * kCellThreads) {
    float px[4], py[4], pz[4], pxr[4], pyd[4], pzn[4], sk[4], c[4], u[4];
    int flags[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = min(i0 + j * kCellThreads, BG::N - 1);
      const int x = x0 - 2 + i % BG::SY, y = y0 - 2 + i / BG::SY % BG::Y, z = z0 - 2 + i / BG::SZ;
      const int cx = min(max(x, 0), G.vx - 1), cy = min(max(y, 0), G.vy - 1), cz = min(max(z, 0), G.vz - 1);
      const int o = cz * plane + cy * pitch + cx;
      const bool nx = cx != G.vx - 1, ny = cy != G.vy - 1, nz = cz != G.vz - 1;
      flags[j] = (cx == x && cy == y && cz == z ? 8 : 0) | (nx ? 1 : 0) | (ny ? 2 : 0) | (nz ? 4 : 0);
      px[j] = V.px_in[o];
      py[j] = V.py_in[o];
      pz[j] = V.pz_in[o];
      pxr[j] = V.px_in[o + (nx ? 1 : 0)];
      pyd[j] = V.py_in[o + (ny ? pitch : 0)];
      pzn[j] = V.pz_in[o + (nz ? plane : 0)];
      sk[j] = V.sink[o];
      c[j] = V.inc[o];
      u[j] = V.label[o];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = i0 + j * kCellThreads;
      if (i >= BG::N) break;
      float d = (px[j] + py[j]) + pz[j];
      if (flags[j] & 1) d = d - pxr[j];
      if (flags[j] & 2) d = d - pyd[j];
      if (flags[j] & 4) d = d - pzn[j];
      const float val = step * (((sk[j] + d) - c[j]) - u[j] * icc);
      g[i] = flags[j] & 8 ? val : 0.0f;
      p[0][i] = px[j];
      p[1][i] = py[j];
      p[2][i] = pz[j];
    }
  }
  __syncthreads();
  // p' = p - (g - g at the lower neighbour), in place (on the box from one
  // below the cell to one above); zero on the low face of its axis and outside
#pragma unroll 2
  for (int i = threadIdx.x; i < BG::N; i += kCellThreads) {
    const int lx = i % BG::SY - 2, ly = i / BG::SY % BG::Y - 2, lz = i / BG::SZ - 2;
    if (lx < -1 || ly < -1 || lz < -1) continue;
    const int x = x0 + lx, y = y0 + ly, z = z0 + lz;
    const bool in = inside(x, y, z);
    const float cur = g[i];
    p[0][i] = in && x ? p[0][i] - (cur - g[i - 1]) : 0.0f;
    p[1][i] = in && y ? p[1][i] - (cur - g[i - BG::SY]) : 0.0f;
    p[2][i] = in && z ? p[2][i] - (cur - g[i - BG::SZ]) : 0.0f;
  }
  __syncthreads();
  // m = |p'| > alpha S ? alpha S / |p'| : 1
#pragma unroll 2
  for (int i = threadIdx.x; i < BM::N; i += kCellThreads) {
    const int lx = i % BM::SY - 1, ly = i / BM::SY % BM::Y - 1, lz = i / BM::SZ - 1;
    const int x = x0 + lx, y = y0 + ly, z = z0 + lz;
    float val = 1.0f;
    if (inside(x, y, z)) {
      const int s = BG::at(lx, ly, lz);
      float up = p[0][s] * p[0][s];
      float dn = x != G.vx - 1 ? p[0][s + 1] * p[0][s + 1] : 0.0f;
      float F = up + dn;
      up = p[1][s] * p[1][s];
      dn = y != G.vy - 1 ? p[1][s + BG::SY] * p[1][s + BG::SY] : 0.0f;
      F = F + (up + dn);
      up = p[2][s] * p[2][s];
      dn = z != G.vz - 1 ? p[2][s + BG::SZ] * p[2][s + BG::SZ] : 0.0f;
      F = F + (up + dn);
      const float h = 0.5f * F;
      const float lim = V.smooth ? V.alpha * V.smooth[z * plane + y * pitch + x] : V.alpha;
      if (!((lim * lim) * (1.0f - 0x1p-20f) - h > 1.0e-36f)) {  // (as in flow_tma_kernel)
        if (!multiplier_unsafe(h, lim)) {
          val = multiplier_fast(h, lim);
        } else {
          const float Fs = sqrtf(h);
          if (Fs > lim) val = lim / Fs;
        }
      }
    }
    m[i] = val;
  }
  __syncthreads();
  // P = (p' / 2) (m + m at the lower neighbour) and its divergence
#pragma unroll
  for (int i = threadIdx.x; i < kCellX * kCellY * kCellZ; i += kCellThreads) {
    const int lx = i % kCellX, ly = i / kCellX % kCellY, lz = i / (kCellX * kCellY);
    const int x = x0 + lx, y = y0 + ly, z = z0 + lz;
    if (!inside(x, y, z)) continue;
    const int s = BG::at(lx, ly, lz), t = BM::at(lx, ly, lz);
    const float mc = m[t];
    const float Px = x ? (p[0][s] * 0.5f) * (mc + m[t - 1]) : 0.0f;
    const float Py = y ? (p[1][s] * 0.5f) * (mc + m[t - BM::SY]) : 0.0f;
    const float Pz = z ? (p[2][s] * 0.5f) * (mc + m[t - BM::SZ]) : 0.0f;
    float d = (Px + Py) + Pz;
    if (x != G.vx - 1) d = d - (p[0][s + 1] * 0.5f) * (m[t + 1] + mc);
    if (y != G.vy - 1) d = d - (p[1][s + BG::SY] * 0.5f) * (m[t + BM::SY] + mc);
    if (z != G.vz - 1) d = d - (p[2][s + BG::SZ] * 0.5f) * (m[t + BM::SZ] + mc);
    const int o = z * plane + y * pitch + x;
    V.px_out[o] = Px;
    V.py_out[o] = Py;
    V.pz_out[o] = Pz;
    V.div[o] = d;
  }
}

// Trees of N <= 8 entries (the root last, entries in post-order).  A thread's
// sinks live in its column of shared memory, where a parent's is found by its
// index; everything else in registers.
constexpr int kSweepCellThreads = 128;
constexpr int kSweepCellMax = 8;

template <int N>
__global__ void __launch_bounds__(kSweepCellThreads)
    sweep_cell_kernel(const TreeTable* __restrict__ table, const Geometry G) {
  constexpr int R = N - 1;  // the root entry
  __shared__ TreeEntry E[N];
  __shared__ float sink[N][kSweepCellThreads];
  dependents_may_launch();
  wait_for_previous_grid();
  for (int i = threadIdx.x; i < (int)(sizeof(E) / 4); i += kSweepCellThreads)
    reinterpret_cast<int*>(E)[i] = reinterpret_cast<const int*>(table->e)[i];
  const float icc = table->icc, cc = table->cc, w0r = table->root_init;
  __syncthreads();
  const int t = threadIdx.x;
  unsigned kmask[N];
#pragma unroll
  for (int e = 0; e < N; ++e) {
    kmask[e] = 0;
#pragma unroll
    for (int k = 0; k < R; ++k)
      if (E[k].parent == e) kmask[e] |= 1u << k;
  }
  for (long long i = (long long)blockIdx.x * kSweepCellThreads + t; i < G.vol;
       i += (long long)gridDim.x * kSweepCellThreads) {
    float d[N], u[N], sc[N];  // divergence, label, old sink (branch) or capacity (leaf)
#pragma unroll
    for (int e = 0; e < R; ++e) {
      d[e] = E[e].div[i];
      u[e] = E[e].label[i];
      sc[e] = (E[e].n_kids ? E[e].sink : E[e].data)[i];
    }
    sc[R] = E[R].sink[i];
#pragma unroll
    for (int e = 0; e < N; ++e) sink[e][t] = sc[e];
#pragma unroll
    for (int e = 0; e < N; ++e) {
      const bool leaf = e != R && E[e].n_kids == 0;
      float v;
      if (leaf) {
        v = (sink[E[e].parent][t] - d[e]) + u[e] * icc;
        v = (v < 0.0f) ? 0.0f : v;
        v = (v > sc[e]) ? sc[e] : v;
      } else {
        float W = e == R ? w0r : 0.0f;
#pragma unroll
        for (int k = 0; k < e; ++k)
          if (kmask[e] >> k & 1u) W = ((W + sc[k]) + d[k]) - u[k] * icc;
        if (e != R) W = ((W + sink[E[e].parent][t]) - d[e]) + u[e] * icc;
        v = W * E[e].inv_kids;
      }
      sc[e] = v;  // the new sink
      sink[e][t] = v;
    }
#pragma unroll
    for (int e = 0; e < R; ++e) {
      E[e].label_out[i] = __saturatef(u[e] + cc * ((sink[E[e].parent][t] - d[e]) - sc[e]));
      E[e].sink_out[i] = sc[e];
    }
    E[R].sink_out[i] = sc[R];
  }
}

}  // namespace hmf
