// hmf_adjoint_flow.cuh -- reverse of the flow step of every non-root vertex
// in one launch, TMA-fed (the fused form of adj_grad .. adj_oldflow in
// hmf_adjoint.cuh, same FP32 operations in the same order).
//
// Per voxel and vertex the reverse needs the state before the iteration
// (three flows, sink, parent sink, label, smoothness) and the adjoints of the
// new flows and of the new divergence, and produces the adjoints of the old
// flows and of the gradient-step values g.  Its stencil chain
//   g -> p' -> (|p|, m, adjoint of m -> F2b) -> q -> gb -> old-flow adjoint
// reaches three voxels to the low side and two to the high side, so a CTA
// owns a 32 x 32 (x, y) window with up to 26 x 27 outputs (the window starts
// four columns low, so that its pairs of columns are 8-byte aligned) and
// marches along z.  A half-warp covers a row (y0-3+row), two neighbouring
// columns (x0-4+2 lane) per lane as one 64-bit register pair: loads and stores
// move 8 bytes and the arithmetic is packed (hmf_f32x2.cuh).  x neighbours are
// the pair's other half or one warp shuffle, y neighbours go through exchange
// rows in shared memory, z neighbours stay in registers.  Beyond the high faces
// p', t and q are zero, so what the reference leaves out there is added as
// zero.  The step of plane k computes g, p' and the total new-flow adjoint t on
// plane k, m / F2b and q's x and z parts on k-1, q's y part on k-2, gb on k-3
// and the old-flow adjoints on k-4, so that all it takes from its neighbours
// was written before its one CTA barrier.  Input planes arrive by
// cp.async.bulk.tensor into mbarrier rings three planes ahead; one thread waits
// for the next step's, before the barrier; every wait is bounded and a time-out
// sets the error flag.  The plane copies are spread over the
// warps' first lanes (one array each, one mbarrier arrival per array), and
// the steady planes of the march -- every stage active, no z boundary near --
// run a copy of the step compiled without those tests.
//
// What bounds it: latency and issue with the 16 warps that its registers and
// rings allow (63 % of the issue slots, DRAM at 31 %).  128^3, 4 leaves, the mean of
// 300 steps: 196 us a launch, against 211 us with one column and two rows per
// thread, scalar arithmetic and the alpha gradient's sum in double.  With two
// barriers per step and a step less per chunk it took 2 to 3 us more (54 % of
// the issue slots); with every thread waiting for its planes 5 us more.
#pragma once

#include <cuda.h>

#include "hmf_async.cuh"
#include "hmf_f32x2.cuh"
#include "hmf_ff.cuh"
#include "hmf_multiplier.cuh"
#include "hmf_types.cuh"

namespace hmf {

constexpr int kAfBoxX = 36;                 // TMA box width (16-byte aligned start, 33 columns used)
constexpr int kAfBoxY = 33;                 // TMA box height (32 rows + the row below for div)
constexpr int kAfPlane = 1216;              // floats per staged plane (36 x 33 padded to 128 bytes)
constexpr int kAfMainArrays = 10;           // px, py, s, c, u, Pbx, Pby, Pbz, dbp, S
constexpr int kAfMainSlots = 3;
constexpr int kAfPzSlots = 4;
// Plane k + kAfMainLead (main ring) and pz of plane k + 1 + kAfPzLead are
// issued in step k after its CTA barrier, when plane k has been read: the
// leads are kAfMainSlots and kAfPzSlots - 1.
constexpr int kAfMainLead = 3;
constexpr int kAfPzLead = 3;
constexpr int kAfRows = 32;                 // window rows, one per half-warp
constexpr int kAfThreads = 16 * kAfRows;    // 512
constexpr int kAfWarps = kAfThreads / 32;
constexpr int kAfX = (kAfRows + 2) * 32;    // one exchange row per window row, plus zero rows -1 and 32
constexpr int kAfXPlanes = 14;              // g, p'y, ty, m, F2b, qy, dbo: two each, by step parity
constexpr int kAfMaxOutX = 26, kAfMaxOutY = 27;
constexpr int kAfSmemBytes =
    (kAfMainSlots * kAfMainArrays + kAfPzSlots) * kAfPlane * 4 + kAfXPlanes * kAfX * 4 + 64;

struct AdjFlowVertex {  // 64-byte aligned through its CUtensorMap members
  CUtensorMap px, py, pz, s, c, u, smooth;  // state before the iteration
  CUtensorMap pb[2][3];                     // [parity][axis] adjoint of the new flows
  CUtensorMap dbp;                          // adjoint of the new divergence
  float* pb_out[2][3];                      // [parity][axis] adjoint of the old flows
  float* gb;                                // adjoint of g
  double* alpha_grad;
  float alpha;
  int has_smooth;
};

struct AdjFlowParams {
  float step, icc;
  float neg_zero;  // -0: the addend of packed multiplications (hmf_f32x2.cuh)
  int parity;      // which Pb set is read (the other is written)
  int n_vertices;  // grid.x = n_vertices * items
  const FlowVolume* vols;
  const FlowItem* items;
  int* error_flag;
  unsigned long long wait_limit_ns;  // bound of every copy wait (kTmaWaitLimitNs unless a caller sets it)
};

__global__ void __launch_bounds__(kAfThreads, 1)
adj_flow_tma_kernel(const AdjFlowVertex* __restrict__ vertices, const AdjFlowParams fp) {
  extern __shared__ __align__(1024) unsigned char af_raw[];
  float* mslots = reinterpret_cast<float*>(af_raw);                      // [3][10][1216]
  float* zslots = mslots + kAfMainSlots * kAfMainArrays * kAfPlane;      // [4][1216]
  float* xp = zslots + kAfPzSlots * kAfPlane;                            // [14][34][32]
  uint64_t* mbars = reinterpret_cast<uint64_t*>(xp + kAfXPlanes * kAfX); // [3]
  uint64_t* zbars = mbars + kAfMainSlots;                                // [4]
  uint64_t* stall_bar = zbars + kAfPzSlots;                              // [1] never completed (a requested stall)
  // exchange rows: *_L is read by the row above it (its y-1 neighbour), *_F by
  // the row below (y+1)
  float* XG_L = xp;
  float* XPPY_F = xp + 2 * kAfX;
  float* XTY_F = xp + 4 * kAfX;
  float* XM_L = xp + 6 * kAfX;
  float* XF_L = xp + 8 * kAfX;
  float* XQY_F = xp + 10 * kAfX;
  float* XD_L = xp + 12 * kAfX;
  __shared__ int abort_cta, stall_cta;
  __shared__ int stop_cta[2];  // by step parity
  __shared__ double red[kAfWarps];
  dependents_may_launch();

  const int nv = fp.n_vertices;
  const FlowItem item = fp.items[blockIdx.x / nv];
  const FlowVolume FV = fp.vols[item.vol];
  const Geometry G = FV.G;
  const AdjFlowVertex* V = vertices + (size_t)item.vol * nv + (blockIdx.x % nv);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned FULL = 0xffffffffu;
  const int ocols = FV.out_x, orows = FV.out_y;
  const int x0 = (item.tile % FV.tiles_x) * ocols;
  const int y0 = (item.tile / FV.tiles_x) * orows;
  const int xs = (x0 / 4) * 4 - 4;        // x0 - 4 rounded down to a multiple of 4 (x0 >= 0, even)
  const int off = (x0 - 4) - xs;           // 0 or 2
  const int col = (lane & 15) * 2, row = warp * 2 + (lane >> 4);
  const int x = x0 - 4 + col, y = y0 - 3 + row;
  const int zs = item.zc * FV.zchunk;
  const int ze = min(zs + FV.zchunk, G.vz);
  const int kstart = max(zs - 3, 0);
  const int kend = ze + 3;
  const int kA_end = min(ze + 1, G.vz - 1);   // last plane whose g is computed
  const int kpz_end = min(ze + 2, G.vz - 1);  // its divergence reads pz of the next plane
  const int par = fp.parity;
  const float step = fp.step, icc = fp.icc;
  const bool has_s = V->has_smooth != 0;
  const int narr = has_s ? 10 : 9;
  const float alpha = V->alpha;
  float* const ox = V->pb_out[par][0];
  float* const oy = V->pb_out[par][1];
  float* const oz = V->pb_out[par][2];
  float* const ogb = V->gb;
  const bool yin = y >= 0 && y < G.vy;
  bool in[2], face_x[2], face_y[2];  // the pair's voxels inside the volume; and off its low x / y face
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    in[j] = yin && x + j >= 0 && x + j < G.vx;
    face_x[j] = in[j] && x + j > 0;
    face_y[j] = in[j] && y > 0;
  }
  // outputs: pairs of columns (ocols is even; the second may be the first
  // padding column, which gets zero)
  const bool own = in[0] && col >= 4 && col < 4 + ocols && row >= 3 && row < 3 + orows;
  const long long rowoff = (long long)y * G.pitch + x;
  const int si = row * kAfBoxX + off + col;  // element in a staged plane
  const int xw = (row + 1) * 32 + col;       // this pair's entry in an exchange row

  wait_for_previous_grid();
  if (threadIdx.x == 0) {
    const int flag = fp.error_flag ? *(volatile int*)fp.error_flag : 0;
    abort_cta = flag & 2;
    stall_cta = take_stall_request(fp.error_flag, flag);
    if (smem_addr(af_raw) & 127) {  // TMA destinations must be 128-byte aligned
      abort_cta = 1;
      if (fp.error_flag) atomicOr(fp.error_flag, 4);
    }
    for (int s = 0; s < kAfMainSlots; ++s) mbar_init(&mbars[s], (unsigned)narr);
    for (int s = 0; s < kAfPzSlots; ++s) mbar_init(&zbars[s], 1);
    mbar_init(stall_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    stop_cta[0] = stop_cta[1] = 0;
  }
  // exchange rows -1 and 32 are read as zeros (never written)
  for (int i = threadIdx.x; i < kAfXPlanes * kAfX; i += kAfThreads) xp[i] = 0.f;
  __syncthreads();
  if (abort_cta) return;

  auto mslot = [&](int p) { return mslots + ((p - kstart) % kAfMainSlots) * (kAfMainArrays * kAfPlane); };
  auto zslot = [&](int p) { return zslots + ((p - kstart) % kAfPzSlots) * kAfPlane; };
  // Array a of plane p into the main ring (px, py, s, c, u, Pb x/y/z, dbp, S):
  // one thread per array, each with its own expect_tx.
  auto main_map = [&](int a) -> const CUtensorMap* {
    return a < 5 ? &V->px + (a < 2 ? a : a + 1) : a < 8 ? &V->pb[par][a - 5] : a == 8 ? &V->dbp : &V->smooth;
  };
  auto issue_main_array = [&](int p, int a, const CUtensorMap* map) {
    uint64_t* bar = &mbars[(p - kstart) % kAfMainSlots];
    mbar_expect_tx(bar, (unsigned)(kAfBoxX * kAfBoxY * 4));
    tma_load_plane(mslot(p) + a * kAfPlane, map, xs, y0 - 3, p, bar);
  };
  const CUtensorMap* const warp_map = main_map(warp < narr ? warp : 0);
  auto issue_pz = [&](int p) {  // one thread
    uint64_t* bar = &zbars[(p - kstart) % kAfPzSlots];
    mbar_expect_tx(bar, (unsigned)(kAfBoxX * kAfBoxY * 4));
    tma_load_plane(zslot(p), &V->pz, xs, y0 - 3, p, bar);
  };
  // Thread 0 alone waits for the planes the next step reads, before the step's
  // CTA barrier (the barrier extends its acquire to every thread).  A wait that
  // runs out raises the step's flag, read by all after its barrier: the CTA
  // leaves the march, drains its copies and reports.
  bool timed_out = false;
  auto wait0 = [&](uint64_t* bar, unsigned parity, int k) {  // thread 0 only
    if (timed_out || mbar_wait_bounded(bar, parity, fp.wait_limit_ns)) return;
    timed_out = true;
    *(volatile int*)&stop_cta[k & 1] = 1;
  };
  int k_stop = -1;  // the step at which the march stopped (-1: it ran to the end)
  auto wait_main0 = [&](int p, int k) {
    wait0(&mbars[(p - kstart) % kAfMainSlots], (unsigned)(((p - kstart) / kAfMainSlots) & 1), k);
  };
  auto wait_pz0 = [&](int p, int k) {
    wait0(&zbars[(p - kstart) % kAfPzSlots], (unsigned)(((p - kstart) / kAfPzSlots) & 1), k);
  };
  // Lane 0 of warp a issues every copy of main-ring array a, lane 0 of the
  // last warp every z-flow copy; each first acquires the one map it uses.
  if (lane == 0) {
    if (warp < narr) {
      tensormap_acquire(warp_map);
      for (int p = kstart; p <= min(kstart + kAfMainLead - 1, kA_end); ++p) issue_main_array(p, warp, warp_map);
    }
    if (warp == kAfWarps - 1) {
      tensormap_acquire(&V->pz);
      for (int p = kstart; p <= min(kstart + kAfPzLead, kpz_end); ++p) issue_pz(p);
    }
  }
  if (threadIdx.x == 0) {
    wait_main0(kstart, kstart);
    wait_pz0(kstart, kstart);
    if (kstart + 1 < G.vz) wait_pz0(kstart + 1, kstart);
    // the failure path on demand: a wait on a barrier that no copy completes
    if (stall_cta) wait0(stall_bar, 0, kstart);
  }
  __syncthreads();

  // A window whose 32 x 32 columns / rows lie inside the volume and off its low
  // faces needs none of the x / y boundary masks; it runs a copy of the march
  // with them folded away.
  const bool interior = x0 - 4 >= 1 && x0 + 27 <= G.vx - 1 && y0 - 3 >= 1 && y0 + 28 <= G.vy - 1;
  FF asum{0.0f, 0.0f};  // alpha gradient (float-float: this part's FP64 rate is 1/64 of its FP32 rate)

  auto march = [&](auto tag) {
    constexpr bool INT = decltype(tag)::value;
    const F2 zero2 = f2(0.f), half2 = f2(0.5f), two2 = f2(2.0f), step2 = f2(step), icc2 = f2(icc), alpha2 = f2(alpha);
    const F2 nz2 = f2(fp.neg_zero);
    auto mul = [&](F2 a, F2 b) { return f2_mul(a, b, nz2); };
    auto left = [&](F2 a) { return f2(__shfl_up_sync(FULL, f2_hi(a), 1, 16), f2_lo(a)); };      // at x - 1
    auto right = [&](F2 a) { return f2(f2_hi(a), __shfl_down_sync(FULL, f2_lo(a), 1, 16)); };  // at x + 1
    auto inside = [&](F2 a) { return INT ? a : f2_mask(a, in[0], in[1]); };
    auto off_x = [&](F2 a) { return INT ? a : f2_mask(a, face_x[0], face_x[1]); };
    auto off_y = [&](F2 a) { return INT ? a : f2_mask(a, face_y[0], face_y[1]); };
    // carries
    F2 gprev = zero2, dbp_prev = zero2;                                                              // plane k-1
    F2 ppx = zero2, ppy = zero2, ppz = zero2, tx = zero2, ty = zero2, tz = zero2, S_c = zero2;       // k-1
    F2 m_prev = f2(1.0f), f_prev = zero2;                                                            // k-2
    F2 qx_d = zero2, qz_d = zero2;                                                                   // q of k-2
    F2 qx_e = zero2, qy_e = zero2, qz_e = zero2;                                                     // q of k-3
    F2 qx_f = zero2, qy_f = zero2, qz_f = zero2;                                                     // q of k-4
    F2 dbo_f = zero2, dbo_ff = zero2;                                                                // k-4, k-5
    F2 pzn_c = zero2;
    bool have_pz = false;
    const float* cur = mslot(kstart);
    const float* zc = zslot(kstart);
    int msi = 0, zsi = 0;                           // ring positions of plane k
    long long go = (long long)(kstart - 3) * G.plane;  // plane offset of gb outputs (plane k-3)
    long long fo = (long long)(kstart - 4) * G.plane;  // ... of old-flow outputs (plane k-4)

    // returns false when the march stops (a copy wait ran out)
    auto zstep = [&](const int k, auto stag) -> bool {
      constexpr bool ST = decltype(stag)::value;  // a steady plane: every stage, no z boundary near
      const bool doA = ST || k <= kA_end;
      const int kc = k - 1;
      const bool doC = ST || (kc >= kstart && kc <= min(ze, G.vz - 1));
      const bool doY = ST || (k - 2 >= kstart && k - 2 <= min(ze, G.vz - 1));
      const int ko = k - 3;
      const bool doE = ST || (ko >= kstart && ko <= ze - 1);
      const int kf = k - 4;
      const bool doF = ST || (kf >= zs && kf < ze);
      const int now = (k & 1) * kAfX + xw, before = ((k & 1) ^ 1) * kAfX + xw;  // exchange rows of this step, of the last

      // ---- stage A: g(k) (kern_CalcGradStep on the recomputed divergence)
      F2 g = zero2, px = zero2, py = zero2, pz = zero2, Pbx = zero2, Pby = zero2, Pbz = zero2, dbp = zero2,
         dbpl = zero2, dbpu = zero2, Sk = zero2;
      if (doA) {
        const bool has_next = ST || k + 1 < G.vz;
        const int znext = zsi + 1 == kAfPzSlots ? 0 : zsi + 1;
        const float* zn = zslots + znext * kAfPlane;
        px = f2_ld(cur + si);
        py = f2_ld(cur + kAfPlane + si);
        pz = (ST || have_pz) ? pzn_c : f2_ld(zc + si);
        const F2 pxr = f2(f2_hi(px), cur[si + 2]);
        const F2 pyd = f2_ld(cur + kAfPlane + si + kAfBoxX);
        const F2 pzn = has_next ? f2_ld(zn + si) : zero2;
        const F2 sk = f2_ld(cur + 2 * kAfPlane + si), c = f2_ld(cur + 3 * kAfPlane + si),
                 u = f2_ld(cur + 4 * kAfPlane + si);
        Pbx = f2_ld(cur + 5 * kAfPlane + si);
        Pby = f2_ld(cur + 6 * kAfPlane + si);
        Pbz = f2_ld(cur + 7 * kAfPlane + si);
        dbp = f2_ld(cur + 8 * kAfPlane + si);
        dbpl = f2(off + col > 0 ? cur[8 * kAfPlane + si - 1] : 0.f, f2_lo(dbp));
        dbpu = row > 0 ? f2_ld(cur + 8 * kAfPlane + si - kAfBoxX) : zero2;
        if (has_s) Sk = f2_ld(cur + 9 * kAfPlane + si);
        F2 d = (px + py) + pz;
        d = d - pxr;
        d = d - pyd;
        d = d - pzn;
        g = mul(step2, ((sk + d) - c) - mul(u, icc2));
        pzn_c = pzn;
        have_pz = has_next;
      }
      f2_st(XG_L + now, g);
      if (threadIdx.x == 0) {  // the planes the next step's stage A reads
        if (k + 1 <= kA_end) wait_main0(k + 1, k);
        if (k + 2 < G.vz && k + 2 <= kpz_end) wait_pz0(k + 2, k);
      }
      __syncthreads();
      if (*(volatile int*)&stop_cta[k & 1]) {
        k_stop = k;
        return false;
      }
      if (lane == 0) {
        if (warp < narr && k + kAfMainLead <= kA_end) issue_main_array(k + kAfMainLead, warp, warp_map);
        if (warp == kAfWarps - 1 && k + 1 + kAfPzLead <= kpz_end) issue_pz(k + 1 + kAfPzLead);
      }

      // ---- stage B: p'(k) (kern_DescentSpatialFlow) and the total adjoint t(k)
      // of the new flows (incoming plus through the new divergence)
      F2 ppx_n = off_x(px - (g - left(g)));
      F2 ppy_n = off_y(py - (g - f2_ld(XG_L + now - 32)));
      F2 ppz_n = inside(pz - (g - gprev));
      F2 tx_n = inside((Pbx + dbp) - dbpl);
      F2 ty_n = inside((Pby + dbp) - dbpu);
      F2 tz_n = inside((Pbz + dbp) - ((ST || k > 0) ? dbp_prev : zero2));
      if (!ST) {
        if (!doA) ppx_n = ppy_n = ppz_n = tx_n = ty_n = tz_n = zero2;
        if (k <= 0) ppz_n = zero2;
      }
      if (doA) {
        gprev = g;
        dbp_prev = dbp;
      }
      const F2 ppy_2 = f2_ld(XPPY_F + now), ty_2 = f2_ld(XTY_F + now);  // this thread's of plane k-2
      f2_st(XPPY_F + now, ppy_n);
      f2_st(XTY_F + now, ty_n);

      // ---- stage C: |p|, m(k-1) and the adjoint of the multiplier -> F2b(k-1)
      F2 m = f2(1.0f), f2b = zero2;
      {
        const F2 pyd = f2_ld(XPPY_F + before + 32);
        const F2 tyd = f2_ld(XTY_F + before + 32);
        const F2 pxr = right(ppx), txr = right(tx);
        F2 f = mul(ppx, ppx) + mul(pxr, pxr);
        f = f + (mul(ppy, ppy) + mul(pyd, pyd));
        f = f + (mul(ppz, ppz) + mul(ppz_n, ppz_n));
        const F2 h = mul(half2, f);
        const F2 lim = has_s ? mul(alpha2, S_c) : alpha2;
        // above 1e-36: |p| <= lim exactly and m = 1 (as in flow_tma_kernel)
        F2 slack = mul(mul(lim, lim), f2(1.0f - 0x1p-20f)) - h;
        if (!INT) slack = f2(in[0] ? f2_lo(slack) : 1.0f, in[1] ? f2_hi(slack) : 1.0f);
        const bool near0 = doC && !(f2_lo(slack) > 1.0e-36f), near1 = doC && !(f2_hi(slack) > 1.0e-36f);
        if (__any_sync(FULL, near0 || near1)) {
          F2 mb2 = mul(mul(tx, half2), ppx);  // (terms of the reference's masked faces are zero: p' is)
          mb2 = zero2 + mb2;
          mb2 = mb2 + mul(mul(txr, half2), pxr);
          mb2 = mb2 + mul(mul(ty, half2), ppy);
          mb2 = mb2 + mul(mul(tyd, half2), pyd);
          mb2 = mb2 + mul(mul(tz, half2), ppz);
          mb2 = mb2 + mul(mul(tz_n, half2), ppz_n);
          float mv[2] = {1.0f, 1.0f}, fv[2] = {0.0f, 0.0f};
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const float hj = j ? f2_hi(h) : f2_lo(h), lj = j ? f2_hi(lim) : f2_lo(lim);
            if (j ? near1 : near0) {
              float Fm, mj;
              if (multiplier_unsafe(hj, lj)) {
                Fm = sqrtf(hj);
                mj = lj / Fm;
              } else {
                mj = multiplier_root(hj, lj, Fm);
              }
              if (Fm > lj) {
                const float mb = j ? f2_hi(mb2) : f2_lo(mb2);
                mv[j] = mj;
                fv[j] = -mb * lj / (4.0f * Fm * Fm * Fm);
                if (own && (j == 0 || in[1]) && (ST || kc >= zs) && kc < ze)
                  ff_add(asum, mb / Fm * (has_s ? (j ? f2_hi(S_c) : f2_lo(S_c)) : 1.0f));
              }
            }
          }
          m = f2(mv[0], mv[1]);
          f2b = f2(fv[0], fv[1]);
        }
        f2_st(XM_L + now, m);
        f2_st(XF_L + now, f2b);
      }

      // ---- stage D: q, the adjoint of p': the x and z parts of plane k-1; the
      // y part, which takes the row above's m, of plane k-2
      F2 qy_n = zero2;
      if (doY) {
        const F2 mup = f2_ld(XM_L + before - 32), fup = f2_ld(XF_L + before - 32);
        qy_n = off_y(mul(mul(ty_2, half2), m_prev + mup) + mul(mul(two2, ppy_2), f_prev + fup));
      }
      F2 qx_n = zero2, qz_n = zero2;
      if (doC) {
        qx_n = off_x(mul(mul(tx, half2), m + left(m)) + mul(mul(two2, ppx), f2b + left(f2b)));
        if (ST || kc > 0) qz_n = inside(mul(mul(tz, half2), m + m_prev) + mul(mul(two2, ppz), f2b + f_prev));
        m_prev = m;
        f_prev = f2b;
      }
      f2_st(XQY_F + now, qy_n);  // plane k-2

      // ---- stage E: gb(k-3), the adjoint of g, and dbo = step * gb
      F2 dbo = zero2;
      {
        const F2 qyd = f2_ld(XQY_F + before + 32);  // plane k-3
        const F2 s3 = (qx_e + qy_e) + qz_e;
        F2 gb = f2(-f2_lo(s3), -f2_hi(s3));
        gb = gb + right(qx_e);
        gb = gb + qyd;
        gb = gb + qz_d;
        if (doE) {
          dbo = inside(mul(step2, gb));
          if (own && (ST || ko >= zs)) f2_st(ogb + (go + rowoff), inside(gb));
        }
        f2_st(XD_L + now, dbo);  // plane k-3
      }

      // ---- stage F: adjoint of the old flows at k-4
      {
        const F2 dup = f2_ld(XD_L + before - 32);  // plane k-4
        const F2 dxl = left(dbo_f);
        if (doF && own) {
          const long long o = fo + rowoff;
          f2_st(ox + o, inside((qx_f + dbo_f) - dxl));
          f2_st(oy + o, inside((qy_f + dbo_f) - dup));
          f2_st(oz + o, inside((qz_f + dbo_f) - ((ST || kf > 0) ? dbo_ff : zero2)));
        }
      }

      // ---- rotate carries and ring positions
      ppx = ppx_n;
      ppy = ppy_n;
      ppz = ppz_n;
      tx = tx_n;
      ty = ty_n;
      tz = tz_n;
      S_c = Sk;
      qx_f = qx_e;
      qy_f = qy_e;
      qz_f = qz_e;
      qx_e = qx_d;
      qy_e = qy_n;
      qz_e = qz_d;
      qx_d = qx_n;
      qz_d = qz_n;
      dbo_ff = dbo_f;
      dbo_f = dbo;
      msi = msi + 1 == kAfMainSlots ? 0 : msi + 1;
      zsi = zsi + 1 == kAfPzSlots ? 0 : zsi + 1;
      cur = mslots + msi * (kAfMainArrays * kAfPlane);
      zc = zslots + zsi * kAfPlane;
      go += G.plane;
      fo += G.plane;
      return true;
    };
    const int k_lo = zs + 5, k_hi = min(ze + 1, G.vz - 2);
    int k = kstart;
    bool go_on = true;
    for (; go_on && k <= kend && k < k_lo; ++k) go_on = zstep(k, BoolTag<false>{});
    for (; go_on && k <= k_hi; ++k) go_on = zstep(k, BoolTag<true>{});
    for (; go_on && k <= kend; ++k) go_on = zstep(k, BoolTag<false>{});
  };
  if (interior) march(BoolTag<true>{});
  else march(BoolTag<false>{});

  // alpha gradient: block sum, one atomic per CTA
  double alpha_sum = (double)asum.hi + (double)asum.lo;
  for (int o = 16; o > 0; o >>= 1) alpha_sum += __shfl_down_sync(FULL, alpha_sum, o);
  if (lane == 0) red[warp] = alpha_sum;
  __syncthreads();
  if (warp == 0) {
    double v = lane < kAfWarps ? red[lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(FULL, v, o);
    if (lane == 0 && v != 0.0) atomicAdd(V->alpha_grad, v);
  }
  if (timed_out && threadIdx.x == 0) {
    if (fp.error_flag) atomicOr(fp.error_flag, 2);
    // Copies still in flight into this CTA's shared memory must land before
    // it exits.  Up to the step before k_stop, ks, the main ring was filled to
    // plane ks + kAfMainLead and the pz ring to ks + 1 + kAfPzLead (the
    // initial issue: kstart - 1 + kAfMainLead, kstart + kAfPzLead), each slot
    // holding at most one pending phase: wait for the last plane issued into
    // each slot, with the default bound.
    const int ks = max(k_stop, kstart) - 1;
    const int l_main = min(max(ks + kAfMainLead, kstart + kAfMainLead - 1), kA_end);
    const int l_pz = min(max(ks + 1 + kAfPzLead, kstart + kAfPzLead), kpz_end);
    for (int p = max(kstart, l_main - kAfMainSlots + 1); p <= l_main; ++p)
      mbar_wait_bounded(&mbars[(p - kstart) % kAfMainSlots], (unsigned)(((p - kstart) / kAfMainSlots) & 1),
                        kTmaWaitLimitNs);
    for (int p = max(kstart, l_pz - kAfPzSlots + 1); p <= l_pz; ++p)
      mbar_wait_bounded(&zbars[(p - kstart) % kAfPzSlots], (unsigned)(((p - kstart) / kAfPzSlots) & 1),
                        kTmaWaitLimitNs);
  }
}

}  // namespace hmf
