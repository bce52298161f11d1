// godunov_tile.cuh -- the level-wide godunov kernel (godunov_fine.f90:5-35,
// godfine1 :486-911 and unsplit, umuscl.f90:22-171) as a tiled sm_100a stencil.
//
// A tile is an aligned box of TX x TY x TZ level-l cells (TX/2 x TY/2 x TZ/2
// octs). One CTA owns one tile, one thread one cell of it:
//   A. gather the (TX+4)(TY+4)(TZ+4) stencil into shared memory as primitive
//      variables. Each 2x2x2 block of the stencil is an existing level-l oct
//      (read from uold), a prolongated coarse cell (interpol_hydro, computed
//      beforehand into the interpolation buffer), or absent (no active oct
//      reads it); plus the refinement flag son(cell)>0 of every cell;
//   B. slopes + MUSCL-Hancock trace: every thread its own cell, whose states at
//      the lower faces stay in registers and at the upper faces go to shared
//      memory, then one cell of the one-cell face slabs around the tile;
//   C. one Riemann problem per face, flux*dt/dx, zeroed where either side is
//      refined (godunov_fine.f90:720-747): every thread the three lower faces
//      of its cell, then the upper faces of the tile's far sides;
//   D. unew += (Fx_l - Fx_r) then y then z for the cells of active octs
//      (godunov_fine.f90:751-792), the lower fluxes from registers;
//   E. the boundary-face fluxes of octs that border an unrefined coarser cell
//      are stored for the deterministic fine-to-coarse correction.
// Every quantity is a pure function of its stencil, so computing each cell
// and face once per tile gives the values the reference computes (redundantly)
// per oct.
//
// What bounds it: instruction issue (FP32-mixed) and the latency of the FP64
// chains (drop-in), so what counts is instructions per cell and CTAs in
// flight. States are packed for 128-bit shared accesses, and only one of a
// face's two states passes through shared memory. The variant that reads the
// scheme at run time differs (kBothStates): it holds every solver and both
// predictors, whose registers are worth more than the shared traffic.
#pragma once
#include <cstdint>
#include <type_traits>

#include "cp_async.cuh"
#include "hydro_core.cuh"

namespace rb {

struct TileArgs {
  const double* __restrict__ uold;      // [5][ncell], device cell layout
  double* __restrict__ unew;            // [5][ncell]
  const int32_t* __restrict__ son;      // [ncell], device cell layout
  const double* __restrict__ interp;    // [5][ninterp*8] prolongated blocks
  const int32_t* __restrict__ tile_blk; // [ntile][NBLK] block codes
  const int32_t* __restrict__ tile_corr_off; // [ntile+1] (null: no correction slots)
  const int32_t* __restrict__ tile_corr;     // [entries][2] (oct in tile | face << 8, slot): the
                                             // faces whose fluxes the fine-to-coarse correction reads
  double* __restrict__ corr_flux;       // [nslot][6][4][5]
  int64_t ncell;
  int64_t ninterp8;                     // ninterp*8 (stride of interp)
  int32_t ncoarse;
  int32_t ntile;
  int32_t has_refined;                  // any son>0 among this level's cells
  int32_t dx_pow2;                      // dx is an exact power of two
  int32_t fused;                        // 1: unew = uold + fluxes (set_unew fused) and
                                        //    CFL partials of the new state; 2: unew = uold +
                                        //    fluxes only (a level without finer octs, whose
                                        //    unew holds no fine-to-coarse correction)
  double dt, dx, inv_dx;
  const double* __restrict__ dt_dev;    // if non-null, dt is read here
  double* __restrict__ partial;         // fused: [ntile][4] (min dt, mass, E, eint)
  const double* __restrict__ gate;      // if non-null and *gate != 0 the launch is a no-op
  double* __restrict__ divu;            // pressure_fix (PF kernels): [ncell] velocity divergence
  double* __restrict__ enew;            //   and internal energy, updated like unew
  double* __restrict__ corr_tmp;        //   [nslot][6][4][2] their correction-face fluxes
  rb_hydro_params hp;
};

// block code: >= 0 oct index (igrid-1); -1 absent; <= -2 interpolation entry (-code-2)
template <int TX, int TY, int TZ>
struct TileGeom {
  // stencil; the row stride is odd, so that the x slabs' column accesses (16
  // bytes per lane) fall into different banks
  static constexpr int SX = TX + 5, SY = TY + 4, SZ = TZ + 4;
  static constexpr int NS = SX * SY * SZ;
  static constexpr int BX = TX / 2 + 2, BY = TY / 2 + 2, BZ = TZ / 2 + 2;
  static constexpr int NBLK = BX * BY * BZ;
  // face-state arrays (per variable)
  static constexpr int NFX = (TX + 1) * TY * TZ;
  static constexpr int NFY = TX * (TY + 1) * TZ;
  static constexpr int NFZ = TX * TY * (TZ + 1);
  static constexpr int NF = NFX + NFY + NFZ;
  static constexpr int NCELL = TX * TY * TZ;
  // one-cell face slabs: lower and upper side of x, y, z; the upper sides'
  // faces are the tile's far faces
  static constexpr int NUX = TY * TZ, NUY = TX * TZ, NUZ = TX * TY;
  static constexpr int NU = NUX + NUY + NUZ;
  static constexpr int NSLAB = 2 * NU;
};

// Stencil cells read by the slopes of types 0, 1, 2, 7 and 8: the tile, its
// one-cell face slabs and their six neighbours. Listed block-major as
// (block << 3 | child): all children of a block with at most one halo
// coordinate, the two inner-layer children of an edge block (two halo
// coordinates), nothing of a corner block.
template <int TX, int TY, int TZ>
constexpr int gather_children(int b, int ch) {
  using G = TileGeom<TX, TY, TZ>;
  const int bx = b % G::BX, by = (b / G::BX) % G::BY, bz = b / (G::BX * G::BY);
  const bool hx = bx == 0 || bx == G::BX - 1, hy = by == 0 || by == G::BY - 1, hz = bz == 0 || bz == G::BZ - 1;
  const int nh = (int)hx + (int)hy + (int)hz;
  if (nh <= 1) return 1;
  if (nh == 3) return 0;
  // inner layer: child 1 of the first block, child 0 of the last
  const int px = ch & 1, py = (ch >> 1) & 1, pz = ch >> 2;
  if (hx && px != (bx == 0 ? 1 : 0)) return 0;
  if (hy && py != (by == 0 ? 1 : 0)) return 0;
  if (hz && pz != (bz == 0 ? 1 : 0)) return 0;
  return 1;
}
template <int TX, int TY, int TZ>
constexpr int gather_count() {
  int n = 0;
  for (int b = 0; b < TileGeom<TX, TY, TZ>::NBLK; b++)
    for (int ch = 0; ch < 8; ch++) n += gather_children<TX, TY, TZ>(b, ch);
  return n;
}
// entry: stencil slot | block << 12 | child << 21 | (cell of the tile) << 24
template <int TX, int TY, int TZ>
constexpr uint32_t gather_entry(int b, int ch) {
  using G = TileGeom<TX, TY, TZ>;
  const int sx = 2 * (b % G::BX) + (ch & 1), sy = 2 * ((b / G::BX) % G::BY) + ((ch >> 1) & 1),
            sz = 2 * (b / (G::BX * G::BY)) + (ch >> 2);
  const bool inner = sx >= 2 && sx < 2 + TX && sy >= 2 && sy < 2 + TY && sz >= 2 && sz < 2 + TZ;
  return (uint32_t)(sx + G::SX * (sy + G::SY * sz)) | (uint32_t)b << 12 | (uint32_t)ch << 21 | (uint32_t)inner << 24;
}
template <int TX, int TY, int TZ>
struct GatherList {
  static constexpr int N = gather_count<TX, TY, TZ>();
  static_assert(TileGeom<TX, TY, TZ>::NS <= 4096 && TileGeom<TX, TY, TZ>::NBLK <= 512, "entry fields");
  uint32_t e[N];
  constexpr GatherList() : e{} {
    int n = 0;
    for (int b = 0; b < TileGeom<TX, TY, TZ>::NBLK; b++)
      for (int ch = 0; ch < 8; ch++)
        if (gather_children<TX, TY, TZ>(b, ch)) e[n++] = gather_entry<TX, TY, TZ>(b, ch);
  }
};
template <int TX, int TY, int TZ>
__device__ const GatherList<TX, TY, TZ> kGatherList{};

// N five-value states in shared memory, packed for 128-bit accesses: float as
// (r,u,v,w) + p, double as (r,u) + (v,w) + p.
template <typename R> struct States;
template <> struct States<float> {
  float4* a;
  float* b;
  static constexpr __host__ __device__ int pad(int n) { return (n + 3) & ~3; }
  static constexpr __host__ __device__ size_t bytes(int n) { return 20 * (size_t)pad(n); }
  __device__ States(unsigned char* base, int n)
      : a(reinterpret_cast<float4*>(base)), b(reinterpret_cast<float*>(base + 16 * (size_t)pad(n))) {}
  __device__ __forceinline__ Prim<float> get(int i) const {
    const float4 x = a[i];
    return Prim<float>{x.x, x.y, x.z, x.w, b[i]};
  }
  __device__ __forceinline__ void put(int i, const Prim<float>& q) {
    a[i] = make_float4(q.r, q.u, q.v, q.w);
    b[i] = q.p;
  }
  __device__ __forceinline__ float& at(int i, int v) {
    return v < 4 ? reinterpret_cast<float*>(a)[4 * i + v] : b[i];
  }
};
template <> struct States<double> {
  double2 *a, *b;
  double* c;
  static constexpr __host__ __device__ int pad(int n) { return (n + 1) & ~1; }
  static constexpr __host__ __device__ size_t bytes(int n) { return 40 * (size_t)pad(n); }
  __device__ States(unsigned char* base, int n)
      : a(reinterpret_cast<double2*>(base)), b(reinterpret_cast<double2*>(base + 16 * (size_t)pad(n))),
        c(reinterpret_cast<double*>(base + 32 * (size_t)pad(n))) {}
  __device__ __forceinline__ Prim<double> get(int i) const {
    const double2 x = a[i], y = b[i];
    return Prim<double>{x.x, x.y, y.x, y.y, c[i]};
  }
  __device__ __forceinline__ void put(int i, const Prim<double>& q) {
    a[i] = make_double2(q.r, q.u);
    b[i] = make_double2(q.v, q.w);
    c[i] = q.p;
  }
  __device__ __forceinline__ double& at(int i, int v) {
    return v < 2 ? reinterpret_cast<double*>(a)[2 * i + v] : v < 4 ? reinterpret_cast<double*>(b)[2 * i + v - 2] : c[i];
  }
};

// The run-time scheme variant passes both states of every face and the lower
// fluxes of a cell through shared memory, traces cells and slab cells as one
// list of items, a direction at a time, and solves the faces as another list,
// through one copy of the predictors and solvers. With the compiled variants'
// layout (15 states, 15 fluxes and six solver copies per thread) the FP64
// variant needed 202-236 registers, spilled 650 bytes at its 128 and took 7.7 ms where
// this takes 4.2 (acoustic, two coarse steps of levels 6-8; slope type 3 8.3
// against 4.9); FP32-mixed slope type 3 2.91 against 2.83 ms, and a level of 512 octs
// 12.3 against 15.2 us.
template <typename R, int RS>
constexpr bool kBothStates = RS == 0;

// dynamic shared memory: the stencil's primitive states, reused for the face
// fluxes once they are traced; the lower cell's state at every face; the
// upper slab's state at the far faces (BOTH: the upper cell's at every face);
// block codes; flags
template <typename R, int TX, int TY, int TZ, bool BOTH>
struct TileSmem {
  using G = TileGeom<TX, TY, TZ>;
  static constexpr size_t Q = 0;
  static constexpr size_t L = (States<R>::bytes(G::NS > G::NF ? G::NS : G::NF) + 15) & ~(size_t)15;
  static constexpr size_t U = L + ((States<R>::bytes(G::NF) + 15) & ~(size_t)15);
  static constexpr int NUP = BOTH ? G::NF : G::NU;
  static constexpr size_t BLK = U + ((States<R>::bytes(NUP) + 15) & ~(size_t)15);
  static constexpr size_t OK = BLK + sizeof(int32_t) * (size_t)G::NBLK;
  static constexpr size_t SIZE = OK + (size_t)((G::NS + 15) & ~15);
};
template <typename R, int TX, int TY, int TZ, bool BOTH>
constexpr size_t tile_smem_bytes() {
  return TileSmem<R, TX, TY, TZ, BOTH>::SIZE;
}

// The FP32 forms for minmod and moncen and the run-time variant hand each
// direction's face states to their place as they are formed; the others store
// them after the trace (FP64 hllc with minmod spills 64 bytes so, 88 the other
// way; FP32-mixed, 8 bytes and none).
template <typename R, int RS, int ST>
constexpr bool kPutEach = kBothStates<R, RS> || (sizeof(R) == 4 && RS != 0 && (ST == 1 || ST == 2));

// Traced face states of one cell from its state q0 and its neighbours in q
// (stencil slot s): sp[d] at the lower, sm[d] at the upper face of direction d,
// for the directions of mask; with kPutEach, handed to put(d, sp, sm).
template <typename R, int TX, int TY, int TZ, int RS, int ST, typename Put>
__device__ __forceinline__ void trace_slot(const States<R>& q, int s, const Consts<R>& c, int slope_type,
                                           const R dtd[3], unsigned mask, Prim<R> sp[3], Prim<R> sm[3], Put&& put) {
  using G = TileGeom<TX, TY, TZ>;
  constexpr int st[3] = {1, G::SX, G::SX * G::SY};
  const Prim<R> q0 = q.get(s);
  if constexpr (sizeof(R) == 4 && RS != 0 && (ST == 1 || ST == 2)) {
    float hd[5][3], h[5];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const Prim<float> a = q.get(s - st[d]), b = q.get(s + st[d]);
      hd[0][d] = hslope<ST>(a.r, q0.r, b.r);
      hd[1][d] = hslope<ST>(a.u, q0.u, b.u);
      hd[2][d] = hslope<ST>(a.v, q0.v, b.v);
      hd[3][d] = hslope<ST>(a.w, q0.w, b.w);
      hd[4][d] = hslope<ST>(a.p, q0.p, b.p);
    }
    half_step(q0, hd, c.gamma, dtd[0], h);
#pragma unroll
    for (int d = 0; d < 3; d++) {
      if (!(mask & (1u << d))) continue;
      float P[5], M[5];
      face_pair(h, hd, d, q0.r, c.smallr, P, M);
      put(d, Prim<float>{P[0], P[1], P[2], P[3], P[4]}, Prim<float>{M[0], M[1], M[2], M[3], M[4]});
    }
  } else {
    R dq[5][3];
    if (slope_type == 0) {
#pragma unroll
      for (int v = 0; v < 5; v++) { dq[v][0] = (R)0; dq[v][1] = (R)0; dq[v][2] = (R)0; }
    } else if (slope_type != 3) {
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const Prim<R> a = q.get(s - st[d]), b = q.get(s + st[d]);
        dq[0][d] = slope1<R>(a.r, q0.r, b.r, slope_type, c.slope_theta);
        dq[1][d] = slope1<R>(a.u, q0.u, b.u, slope_type, c.slope_theta);
        dq[2][d] = slope1<R>(a.v, q0.v, b.v, slope_type, c.slope_theta);
        dq[3][d] = slope1<R>(a.w, q0.w, b.w, slope_type, c.slope_theta);
        dq[4][d] = slope1<R>(a.p, q0.p, b.p, slope_type, c.slope_theta);
      }
    } else {
      // positivity-preserving multidimensional slope (umuscl.f90:1328-1392)
      const R half = (R)0.5, one = (R)1, zero = (R)0;
      const R qc[5] = {q0.r, q0.u, q0.v, q0.w, q0.p};
      R vmin[5], vmax[5];
      bool first = true;
      for (int kk = -1; kk <= 1; kk++)
        for (int ii = -1; ii <= 1; ii++)
          for (int jj = -1; jj <= 1; jj++) {
            const Prim<R> n = q.get(s + ii + G::SX * (jj + G::SY * kk));
            const R d[5] = {n.r - qc[0], n.u - qc[1], n.v - qc[2], n.w - qc[3], n.p - qc[4]};
#pragma unroll
            for (int v = 0; v < 5; v++) {
              vmin[v] = first ? d[v] : fmn(vmin[v], d[v]);
              vmax[v] = first ? d[v] : fmx(vmax[v], d[v]);
            }
            first = false;
          }
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const Prim<R> a = q.get(s - st[d]), b = q.get(s + st[d]);
        dq[0][d] = half * (b.r - a.r);
        dq[1][d] = half * (b.u - a.u);
        dq[2][d] = half * (b.v - a.v);
        dq[3][d] = half * (b.w - a.w);
        dq[4][d] = half * (b.p - a.p);
      }
#pragma unroll
      for (int v = 0; v < 5; v++) {
        const R dff = half * ((R)fabs(dq[v][0]) + (R)fabs(dq[v][1]) + (R)fabs(dq[v][2]));
        R slop;
        if (dff > zero) slop = fmn(one, fmn((R)fabs(vmin[v]), (R)fabs(vmax[v])) / dff);
        else slop = one;
        dq[v][0] = slop * dq[v][0]; dq[v][1] = slop * dq[v][1]; dq[v][2] = slop * dq[v][2];
      }
    }
    if constexpr (kBothStates<R, RS>) {
      // a direction at a time: the two predictors meet with one pair of states live, not three
#pragma unroll
      for (int d = 0; d < 3; d++) {
        if (!(mask & (1u << d))) continue;
        trace_sel<R, RS, ST>(q0, dq, c, dtd, sp, sm, 1u << d);
        put(d, sp[d], sm[d]);
      }
    } else {
      trace_sel<R, RS, ST>(q0, dq, c, dtd, sp, sm, mask);
    }
  }
}

// A direction known at compile time, as an argument.
template <int D>
struct Axis {
  static constexpr int value = D;
  __host__ __device__ constexpr operator int() const { return D; }
};

// RS (Riemann solver) and ST (slope type) fix the scheme at compile time;
// RS = 0 / ST = -1 read it from a.hp at run time. PF: pressure_fix, the
// velocity-divergence and internal-energy fluxes of every face (umuscl.f90
// cmpflxm's tmp, :845-849) update a.divu and a.enew beside unew
// (godunov_fine.f90:735-744, 775-789). MINB: CTAs per SM the registers are
// bounded for.
template <typename R, int TX, int TY, int TZ, int NT, int MINB, int RS, int ST, bool PF = false>
__global__ void __launch_bounds__(NT, MINB) godunov_tile_kernel(const __grid_constant__ TileArgs a) {
  using G = TileGeom<TX, TY, TZ>;
  constexpr bool kBoth = kBothStates<R, RS>;
  using M = TileSmem<R, TX, TY, TZ, kBoth>;
  constexpr int SX = G::SX, SY = G::SY;
  constexpr int BX = G::BX, BY = G::BY, NBLK = G::NBLK, NCELL = G::NCELL;
  constexpr int NFX = G::NFX, NFY = G::NFY, NF = G::NF;
  static_assert(NCELL <= NT, "one thread per cell");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  States<R> q(smem_raw + M::Q, G::NS);       // stencil
  States<R> F(smem_raw + M::Q, NF);          // fluxes, once the stencil is traced
  States<R> Ls(smem_raw + M::L, NF);         // lower cell's state at a face
  States<R> Us(smem_raw + M::U, M::NUP);     // upper slab's state at a far face (kBoth: upper cell's at a face)
  int32_t* blk = reinterpret_cast<int32_t*>(smem_raw + M::BLK);
  unsigned char* okf = smem_raw + M::OK;

  const int tile = blockIdx.x;
  if (tile >= a.ntile) return;
  const int tid = threadIdx.x;
  const Consts<R> c = make_consts<R>(a.hp);
  const int64_t ncell = a.ncell;

  constexpr int NOCT = (TX / 2) * (TY / 2) * (TZ / 2);
  __shared__ int32_t corr_range[2];
  __shared__ int32_t corr_ent[2 * 6 * NOCT];
  // the gate (the device scheduler's end-of-run flag) is read together with
  // the tile's codes, so that the two loads overlap; every thread reads the
  // same value, so the return is uniform and precedes the barrier
  const double gate = a.gate != nullptr ? *a.gate : 0.0;
  for (int i = tid; i < NBLK; i += NT) blk[i] = a.tile_blk[(int64_t)tile * NBLK + i];
  if (a.tile_corr_off != nullptr && tid < 2) corr_range[tid] = a.tile_corr_off[tile + tid];
  if (gate != 0.0) return;
  __syncthreads();

  // the tile's correction-face entries are copied to shared memory while the
  // tile is computed (they are read at the end)
  if (a.tile_corr_off != nullptr)
    for (int i = tid; i < 2 * (corr_range[1] - corr_range[0]); i += NT)
      cp_async4(corr_ent + i, a.tile_corr + 2 * corr_range[0] + i);
  cp_async_commit();

  // ---- A. gather + ctoprim ------------------------------------------------
  const int slope_type = ST >= 0 ? ST % 10 : a.hp.slope_type;
  // the 27-point slopes and the corner divergence of difmag read the edge and
  // corner cells of the stencil too
  const bool full_gather = slope_type == 3 || (RS == 0 && a.hp.difmag > 0.0);
  // one stencil cell: its raw state is loaded by gather_cell and converted by
  // put_cell (the listed gather keeps the loads of two cells in flight
  // before their conversion). Blocks coded -1 are read by no present cell:
  // only their flags are set.
  auto gather_cell = [&](uint32_t e, double u[5], int& code, int& sonv) {
    code = blk[(e >> 12) & 511];
    const int ch = (e >> 21) & 7;
    sonv = 0;
    // L2-only loads: the tile reads each stencil cell once, and leaving L1
    // to the loads in flight lets more of them be outstanding
    if (code >= 0) {
      const int64_t dc = (int64_t)a.ncoarse + (int64_t)code * 8 + ch;
#pragma unroll
      for (int v = 0; v < 5; v++) u[v] = __ldcg(a.uold + v * ncell + dc);
      if (a.has_refined) sonv = __ldcg(a.son + dc);
    } else if (code <= -2) {
      const int64_t i = (int64_t)(-code - 2) * 8 + ch;
#pragma unroll
      for (int v = 0; v < 5; v++) u[v] = __ldcg(a.interp + v * a.ninterp8 + i);
    }
  };
  auto put_cell = [&](uint32_t e, const double u[5], int code, int sonv) {
    const int s = e & 4095;
    // okf bit 0: the cell is refined (its faces carry no flux); bit 1: a
    // tile-interior cell of a present oct (its faces and update are used)
    okf[s] = (unsigned char)((sonv > 0 ? 1 : 0) | ((e >> 24) && code >= 0 ? 2 : 0));
    if (code != -1) q.put(s, ctoprim_cell<R>(u, a.hp));
  };
  if (!full_gather) {
    using GL = GatherList<TX, TY, TZ>;
    constexpr int NG = GL::N;
    constexpr int PER = (NG + NT - 1) / NT;
    constexpr int NB = PER < 2 ? PER : 2;
    for (int j0 = 0; j0 < PER; j0 += NB) {
      double u[NB][5];
      uint32_t e[NB];
      int code[NB], sonv[NB];
#pragma unroll
      for (int j = 0; j < NB; j++) {
        const int it = tid + (j0 + j) * NT;
        e[j] = ~0u;
        if (j0 + j < PER && it < NG) {
          e[j] = __ldg(&kGatherList<TX, TY, TZ>.e[it]);
          gather_cell(e[j], u[j], code[j], sonv[j]);
        }
      }
#pragma unroll
      for (int j = 0; j < NB; j++)
        if (e[j] != ~0u) put_cell(e[j], u[j], code[j], sonv[j]);
    }
  } else {
    // every cell of the stencil
    for (int it = tid; it < NBLK * 8; it += NT) {
      const int b = it >> 3, ch = it & 7;
      const int sx = 2 * (b % BX) + (ch & 1), sy = 2 * ((b / BX) % BY) + ((ch >> 1) & 1), sz = 2 * (b / (BX * BY)) + (ch >> 2);
      const bool inner = sx >= 2 && sx < 2 + TX && sy >= 2 && sy < 2 + TY && sz >= 2 && sz < 2 + TZ;
      const uint32_t e = (uint32_t)(sx + SX * (sy + SY * sz)) | (uint32_t)b << 12 | (uint32_t)ch << 21 | (uint32_t)inner << 24;
      double u[5];
      int code, sonv;
      gather_cell(e, u, code, sonv);
      put_cell(e, u, code, sonv);
    }
  }
  __syncthreads();

  // ---- B. slopes + trace ----------------------------------------------------
  const double dt = a.dt_dev ? *a.dt_dev : a.dt;
  const R dtdx = (R)(dt / a.dx);  // trace3d.f90 dtdx = dt/dx (dx=dy=dz)
  const R dtd[3] = {dtdx, dtdx, dtdx};
  // this thread's cell; x fastest, so that a quarter warp's 16-byte shared
  // accesses are consecutive and a warp's global rows whole 32-byte sectors
  const bool own = tid < NCELL;
  const int x = tid % TX, y = (tid / TX) % TY, z = (tid / (TX * TY)) % TZ;
  const int s_own = (x + 2) + SX * ((y + 2) + SY * (z + 2));
  const int code_own = own ? blk[(x / 2 + 1) + BX * ((y / 2 + 1) + BY * (z / 2 + 1))] : -1;
  // lower faces of the own cell
  const int fx0 = x + (TX + 1) * (y + TY * z);
  const int fy0 = NFX + x + TX * (y + (TY + 1) * z);
  const int fz0 = NFX + NFY + x + TX * (y + TY * z);
  // present(s): the tile-interior cell belongs to an oct of this level
  // (its update and its faces are used; bit 1 of okf). A block coded -1 is
  // absent and not a stencil source of any present oct, so no face touching
  // it is used.
  // A face on a tile's side is solved by both tiles and must get one flux.
  // FP64 code is never contracted and the FP32 forms of hydro_core.cuh spell
  // their contraction out, so any copy of them rounds alike; the other FP32
  // schemes go through one instance of the trace (own cell j = 0, then the
  // slab cells) and one of the solver (PLMDE: per direction), as loops that are
  // not unrolled (9 % of a Sedov run where it is not needed).
  constexpr bool kOneSite = sizeof(R) == 4 && !(RS != 0 && (ST == 1 || ST == 2));
  Prim<R> P[3];
  // kBoth: cells and slab cells are one list of items
  constexpr int NJ = kBoth ? (NCELL + G::NSLAB + NT - 1) / NT : 1 + (G::NSLAB + NT - 1) / NT;
#pragma unroll (kOneSite ? 1 : 2)
  for (int j = 0; j < NJ; j++) {
    int s = s_own, d = 0, f = 0, r = 0, side = 0;  // slab: slot, direction, face towards the tile
    bool live = code_own != -1;
    unsigned mask = 7u;
    const bool cell = kBoth ? tid + j * NT < NCELL : j == 0;
    if (!cell) {
      const int it = kBoth ? tid + j * NT - NCELL : tid + (j - 1) * NT;
      if (it >= G::NSLAB) break;
      side = it >= G::NU; r = side ? it - G::NU : it;
      if (r < G::NUX) {
        const int yy = r % TY, zz = r / TY;
        d = 0; s = (side ? TX + 2 : 1) + SX * ((yy + 2) + SY * (zz + 2)); f = (TX + 1) * (yy + TY * zz);
      } else if (r < G::NUX + G::NUY) {
        const int k = r - G::NUX, xx = k % TX, zz = k / TX;
        d = 1; s = (xx + 2) + SX * ((side ? TY + 2 : 1) + SY * (zz + 2)); f = NFX + xx + TX * (TY + 1) * zz;
      } else {
        const int k = r - G::NUX - G::NUY, xx = k % TX, yy = k / TX;
        d = 2; s = (xx + 2) + SX * ((yy + 2) + SY * (side ? TZ + 2 : 1)); f = NFX + NFY + xx + TX * yy;
      }
      const int step = d == 0 ? 1 : d == 1 ? SX : SX * SY;
      live = (okf[side ? s - step : s + step] & 2) != 0;
      mask = 1u << d;
    }
    if (!live) continue;
    auto put = [&](int k, const Prim<R>& sp, const Prim<R>& sm) {
      const int far = k == 0 ? TX : k == 1 ? TX * TY : TX * TY * TZ;  // from a line's first face to its last
      if (cell) {
        const int fl = k == 0 ? fx0 : k == 1 ? fy0 : fz0;
        if (kBoth) Us.put(fl, sp);
        else P[k] = sp;
        Ls.put(fl + (k == 0 ? 1 : k == 1 ? TX : TX * TY), sm);
      } else if (side) {  // upper slab: the right state of its face
        Us.put(kBoth ? f + far : r, sp);
      } else {            // lower slab: the left state
        Ls.put(f, sm);
      }
    };
    Prim<R> sp[3], sm[3];
    trace_slot<R, TX, TY, TZ, RS, ST>(q, s, c, slope_type, dtd, mask, sp, sm, put);
    if constexpr (!kPutEach<R, RS, ST>) {
      if (cell) {
#pragma unroll
        for (int k = 0; k < 3; k++) P[k] = sp[k];
        Ls.put(fx0 + 1, sm[0]);
        Ls.put(fy0 + TX, sm[1]);
        Ls.put(fz0 + TX * TY, sm[2]);
      } else if (side) {
        if (d == 0) Us.put(r, sp[0]);
        else if (d == 1) Us.put(r, sp[1]);
        else Us.put(r, sp[2]);
      } else {
        if (d == 0) Ls.put(f, sm[0]);
        else if (d == 1) Ls.put(f, sm[1]);
        else Ls.put(f, sm[2]);
      }
    }
  }
  // difmag > 0 (run-time scheme variant): cmpdivu (uplmde.f90:702-764), the
  // velocity divergence at the cell corners (x-1/2, y-1/2, z-1/2) of the tile,
  // x in 0..TX etc., from the primitive velocities, before phase C reuses q
  constexpr int CXN = TX + 1, CYN = TY + 1, NCORN = (TX + 1) * (TY + 1) * (TZ + 1);
  R* cdiv = nullptr;
  if constexpr (RS == 0) {
    __shared__ R cdiv_s[NCORN];
    cdiv = cdiv_s;
    if (a.hp.difmag > 0.0) {
      const R quarter = (R)0.5 * (R)0.5;
      const R fxd = (R)(quarter / (R)a.dx), fyd = fxd, fzd = fxd;
      for (int it = tid; it < NCORN; it += NT) {
        const int cx = it % CXN, cy = (it / CXN) % CYN, cz = it / (CXN * CYN);
        auto Q = [&](int ox, int oy, int oz, int v) {
          return q.at((cx + ox + 2) + SX * ((cy + oy + 2) + SY * (cz + oz + 2)), v);
        };
        R ux = (R)0, vy = (R)0, wz = (R)0;
        ux = ux + fxd * (Q(0, 0, 0, 1) - Q(-1, 0, 0, 1));
        ux = ux + fxd * (Q(0, -1, 0, 1) - Q(-1, -1, 0, 1));
        vy = vy + fyd * (Q(0, 0, 0, 2) - Q(0, -1, 0, 2) + Q(-1, 0, 0, 2) - Q(-1, -1, 0, 2));
        ux = ux + fxd * (Q(0, 0, -1, 1) - Q(-1, 0, -1, 1) + Q(0, -1, -1, 1) - Q(-1, -1, -1, 1));
        vy = vy + fyd * (Q(0, 0, -1, 2) - Q(0, -1, -1, 2) + Q(-1, 0, -1, 2) - Q(-1, -1, -1, 2));
        wz = wz + fzd * (Q(0, 0, 0, 3) - Q(0, 0, -1, 3) + Q(0, -1, 0, 3) - Q(0, -1, -1, 3) + Q(-1, 0, 0, 3) -
                         Q(-1, 0, -1, 3) + Q(-1, -1, 0, 3) - Q(-1, -1, -1, 3));
        cdiv[it] = ux + vy + wz;
      }
    }
  }
  __syncthreads();

  // ---- C. Riemann fluxes (flux buffer aliases q) ------------------------------
  // raw (conservative) state of stencil cell (sx, sy, sz), as phase A gathered it
  auto raw_cell = [&](int sx, int sy, int sz, double u[5]) {
    const int b = (sx >> 1) + BX * ((sy >> 1) + BY * (sz >> 1));
    const int ch = (sx & 1) + 2 * (sy & 1) + 4 * (sz & 1);
    const int code = blk[b];
    if (code >= 0) {
      const int64_t dc = (int64_t)a.ncoarse + (int64_t)code * 8 + ch;
      for (int v = 0; v < 5; v++) u[v] = __ldcg(a.uold + v * ncell + dc);
    } else if (code <= -2) {
      const int64_t e = (int64_t)(-code - 2) * 8 + ch;
      for (int v = 0; v < 5; v++) u[v] = __ldcg(a.interp + v * a.ninterp8 + e);
    } else {
      for (int v = 0; v < 5; v++) u[v] = 0.0;
    }
  };
  const float smallc2 = (float)c.smallc * (float)c.smallc;
  auto scaled = [&](R v) -> R {
    if (sizeof(R) == 8) {
      // flux = fx*dt/dx, evaluated as (fx*dt)/dx (umuscl.f90:101-163);
      // division by an exact power of two equals the multiplication
      const double t = (double)v * dt;
      return (R)(a.dx_pow2 ? t * a.inv_dx : t / a.dx);
    }
    return v * dtdx;
  };
  // The flux through face f between cell (cx, cy, cz) and its lower
  // neighbour along D, from the states L and Rr: into F (and tmp, with
  // pressure_fix, into Ls[f], which only this thread reads and has read).
  auto face_flux = [&](auto dir, int f, int cx, int cy, int cz, const Prim<R>& L, const Prim<R>& Rr, int fl,
                       Prim<R>& out, R tmp[2]) {
    const int D = dir;
    // refined interface: either neighbour cell refined -> zero flux
    const bool zero_face = (fl & 1) != 0;
    R ql[5], qr[5], fg[6], fo[5];
    to_face(L, D, ql);
    to_face(Rr, D, qr);
    if constexpr (sizeof(R) == 4 && RS != 0 && (ST == 1 || ST == 2)) {
      riemann_f32<RS, PF>(ql, qr, c, smallc2, dtdx, fg);
      from_face(fg, D, fo);
      if (PF) tmp[1] = zero_face ? (R)0 : fg[5];
    } else {
      riemann_sel<R, RS>(ql, qr, c, fg);
      from_face(fg, D, fo);
#pragma unroll
      for (int v = 0; v < 5; v++) fo[v] = scaled(fo[v]);
      if (PF) tmp[1] = zero_face ? (R)0 : scaled(fg[5]);
    }
    if (PF) tmp[0] = zero_face ? (R)0 : scaled((R)0.5 * (ql[1] + qr[1]));
    if (RS == 0 && a.hp.difmag > 0.0) {
      // consup (uplmde.f90:769-866): + dt*difmag*min(0, div1)*(u_R - u_L)
      // with div1 the mean of the face's four corner divergences, added
      // before the refined-face zeroing
      const R quarter = (R)0.5 * (R)0.5;
      auto DV = [&](int ix, int iy, int iz) { return cdiv[ix + CXN * (iy + CYN * iz)]; };
      R div1;
      if (D == 0) {
        div1 = quarter * DV(cx, cy, cz);
        div1 = div1 + quarter * DV(cx, cy + 1, cz);
        div1 = div1 + quarter * (DV(cx, cy, cz + 1) + DV(cx, cy + 1, cz + 1));
      } else if (D == 1) {
        div1 = (R)0;
        div1 = div1 + quarter * (DV(cx, cy, cz) + DV(cx + 1, cy, cz));
        div1 = div1 + quarter * (DV(cx, cy, cz + 1) + DV(cx + 1, cy, cz + 1));
      } else {
        div1 = quarter * (DV(cx, cy, cz) + DV(cx + 1, cy, cz) + DV(cx, cy + 1, cz) + DV(cx + 1, cy + 1, cz));
      }
      div1 = (R)a.hp.difmag * fmn((R)0, div1);
      double ul[5], ur[5];
      raw_cell(cx + 2 - (D == 0), cy + 2 - (D == 1), cz + 2 - (D == 2), ul);
      raw_cell(cx + 2, cy + 2, cz + 2, ur);
#pragma unroll
      for (int v = 0; v < 5; v++) {
        const R t = sizeof(R) == 8 ? (R)((double)(dt * (double)div1) * (ur[v] - ul[v]))
                                   : (R)(dt * (double)div1 * (ur[v] - ul[v]));
        fo[v] = fo[v] + t;
      }
    }
    if (zero_face) {
#pragma unroll
      for (int v = 0; v < 5; v++) fo[v] = (R)0;
    }
    out = Prim<R>{fo[0], fo[1], fo[2], fo[3], fo[4]};
    F.put(f, out);
    if (PF) {
      Ls.at(f, 0) = tmp[0];
      Ls.at(f, 1) = tmp[1];
    }
  };
  // Per direction: the lower face of the own cell (j = 0), then the far faces,
  // whose three groups go to different threads. A face is used only when one
  // of its two cells is a present cell.
  Prim<R> flo[3];    // fluxes through the own cell's lower faces
  R tlo[3][2] = {{(R)0, (R)0}, {(R)0, (R)0}, {(R)0, (R)0}};
  auto dir_faces = [&](auto dir, int f_own, int j0, int j1, int r0, int nu, int n1) {
    constexpr int D = decltype(dir)::value;
    constexpr int step = D == 0 ? 1 : D == 1 ? SX : SX * SY;
    // the far faces' threads start at r0 modulo the block, so that the three
    // directions load different warps
#pragma unroll 1
    for (int j = j0; j < j1; j++) {
      int f = f_own, cx = x, cy = y, cz = z, r = 0;
      if (j == 0) {
        if (!own) continue;
      } else {
        r = (tid + NT - r0 % NT) % NT + (j - 1) * NT;
        if (r >= nu) break;
        const int k0 = r % n1, k1 = r / n1;
        if (D == 0) { cx = TX; cy = k0; cz = k1; f = TX + (TX + 1) * (cy + TY * cz); }
        else if (D == 1) { cx = k0; cy = TY; cz = k1; f = NFX + cx + TX * (TY + (TY + 1) * cz); }
        else { cx = k0; cy = k1; cz = TZ; f = NFX + NFY + cx + TX * (cy + TY * TZ); }
      }
      const int s = (cx + 2) + SX * ((cy + 2) + SY * (cz + 2));
      const int fl = okf[s] | okf[s - step];
      if (!(fl & 2)) continue;
      Prim<R> fo;
      R t[2];
      face_flux(dir, f, cx, cy, cz, Ls.get(f), j == 0 ? P[D] : Us.get(r0 + r), fl, fo, t);
      if (j == 0) {
        flo[D] = fo;
        if (PF) { tlo[D][0] = t[0]; tlo[D][1] = t[1]; }
      }
    }
  };
  // the passes [j0, j1) of every direction
  auto faces = [&](int j0, int j1) {
    constexpr Axis<0> DX{};
    constexpr Axis<1> DY{};
    constexpr Axis<2> DZ{};
    dir_faces(DX, fx0, j0, min(j1, 1 + (G::NUX + NT - 1) / NT), 0, G::NUX, TY);
    dir_faces(DY, fy0, j0, min(j1, 1 + (G::NUY + NT - 1) / NT), G::NUX, G::NUY, TX);
    dir_faces(DZ, fz0, j0, min(j1, 1 + (G::NUZ + NT - 1) / NT), G::NUX + G::NUY, G::NUZ, TX);
  };
  if constexpr (kBoth) {
    // every face on its own, through one copy of the solvers
#pragma unroll 1
    for (int f = tid; f < NF; f += NT) {
      int d, cx, cy, cz;
      if (f < NFX) { d = 0; cx = f % (TX + 1); cy = (f / (TX + 1)) % TY; cz = f / ((TX + 1) * TY); }
      else if (f < NFX + NFY) { const int r = f - NFX; d = 1; cx = r % TX; cy = (r / TX) % (TY + 1); cz = r / (TX * (TY + 1)); }
      else { const int r = f - NFX - NFY; d = 2; cx = r % TX; cy = (r / TX) % TY; cz = r / (TX * TY); }
      const int s = (cx + 2) + SX * ((cy + 2) + SY * (cz + 2));
      const int fl = okf[s] | okf[s - (d == 0 ? 1 : d == 1 ? SX : SX * SY)];
      if (!(fl & 2)) continue;
      Prim<R> fo;
      R t[2];
      face_flux(d, f, cx, cy, cz, Ls.get(f), Us.get(f), fl, fo, t);
    }
  } else if constexpr (kOneSite) {
    faces(0, 1 << 20);
  } else {
    faces(0, 1);        // straight-line code: the three solves overlap
    faces(1, 1 << 20);
  }
  cp_async_wait<0>();  // this thread's correction entries (E)
  __syncthreads();

  // ---- D. conservative update of active octs ----------------------------------
  double smax = 0.0, mass = 0.0, etot = 0.0, eint = 0.0;
  if (code_own >= 0) {
    const int ch = (x & 1) + 2 * (y & 1) + 4 * (z & 1);
    const int64_t dc = (int64_t)a.ncoarse + (int64_t)code_own * 8 + ch;
    if (kBoth) {
      flo[0] = F.get(fx0); flo[1] = F.get(fy0); flo[2] = F.get(fz0);
      if (PF) {
        tlo[0][0] = Ls.at(fx0, 0); tlo[0][1] = Ls.at(fx0, 1);
        tlo[1][0] = Ls.at(fy0, 0); tlo[1][1] = Ls.at(fy0, 1);
        tlo[2][0] = Ls.at(fz0, 0); tlo[2][1] = Ls.at(fz0, 1);
      }
    }
    const Prim<R> fxr = F.get(fx0 + 1), fyr = F.get(fy0 + TX), fzr = F.get(fz0 + TX * TY);
    const R fl[3][5] = {{flo[0].r, flo[0].u, flo[0].v, flo[0].w, flo[0].p},
                        {flo[1].r, flo[1].u, flo[1].v, flo[1].w, flo[1].p},
                        {flo[2].r, flo[2].u, flo[2].v, flo[2].w, flo[2].p}};
    const R fr[3][5] = {{fxr.r, fxr.u, fxr.v, fxr.w, fxr.p},
                        {fyr.r, fyr.u, fyr.v, fyr.w, fyr.p},
                        {fzr.r, fzr.u, fzr.v, fzr.w, fzr.p}};
    double unv[5];
#pragma unroll
    for (int v = 0; v < 5; v++) unv[v] = a.fused ? __ldcg(a.uold + v * ncell + dc) : a.unew[v * ncell + dc];  // set_unew's value
    double dv = 0.0, en = 0.0;
    if (PF) {
      // divu, then enew, each x then y then z, as unew (the fused form
      // starts them from set_unew's values: 0 and the internal energy of uold)
      if (a.fused) {
        const double dd = fmx(unv[0], a.hp.smallr);
        const double uu = unv[1] / dd, vv = unv[2] / dd, ww = unv[3] / dd;
        en = unv[4] - 0.5 * dd * (uu * uu + vv * vv + ww * ww);
      } else {
        dv = a.divu[dc];
        en = a.enew[dc];
      }
    }
#pragma unroll
    for (int v = 0; v < 5; v++) {
      double un = unv[v];
      un = un + ((double)fl[0][v] - (double)fr[0][v]);
      un = un + ((double)fl[1][v] - (double)fr[1][v]);
      un = un + ((double)fl[2][v] - (double)fr[2][v]);
      a.unew[v * ncell + dc] = un;
      unv[v] = un;
    }
    if (PF) {
      dv = dv + ((double)tlo[0][0] - (double)Ls.at(fx0 + 1, 0));
      dv = dv + ((double)tlo[1][0] - (double)Ls.at(fy0 + TX, 0));
      dv = dv + ((double)tlo[2][0] - (double)Ls.at(fz0 + TX * TY, 0));
      en = en + ((double)tlo[0][1] - (double)Ls.at(fx0 + 1, 1));
      en = en + ((double)tlo[1][1] - (double)Ls.at(fy0 + TX, 1));
      en = en + ((double)tlo[2][1] - (double)Ls.at(fz0 + TX * TY, 1));
      a.divu[dc] = dv;
      a.enew[dc] = en;
    }
    if (a.fused == 1) {
      // courant_fine on the updated state (the next step's CFL condition);
      // the level minimum of dt_cell is dt_cell(maximum wave speed)
      const double vol = a.dx * a.dx * a.dx;
      const double ir = 1.0 / fmx(unv[0], a.hp.smallr);
      mass = mass + unv[0] * vol;
      etot = etot + unv[4] * vol;
      eint = eint + (unv[4] - 0.5 * (unv[1] * unv[1] + unv[2] * unv[2] + unv[3] * unv[3]) * ir) * vol;
      smax = fmx(smax, sizeof(R) == 8 ? cfl_speed(unv, a.hp) : cfl_speed_fast(unv, a.hp));
    }
  }
  if (a.fused == 1) {
    __shared__ double red[4][NT / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      smax = fmx(smax, __shfl_xor_sync(0xffffffffu, smax, o));
      mass += __shfl_xor_sync(0xffffffffu, mass, o);
      etot += __shfl_xor_sync(0xffffffffu, etot, o);
      eint += __shfl_xor_sync(0xffffffffu, eint, o);
    }
    if ((tid & 31) == 0) { red[0][tid >> 5] = smax; red[1][tid >> 5] = mass; red[2][tid >> 5] = etot; red[3][tid >> 5] = eint; }
    __syncthreads();
    if (tid == 0) {
      for (int k = 1; k < NT / 32; k++) { smax = fmx(smax, red[0][k]); mass += red[1][k]; etot += red[2][k]; eint += red[3][k]; }
      a.partial[(int64_t)tile * 4 + 0] = smax > 0.0 ? cfl_dt_from_speed(smax, a.dx, a.hp.courant_factor) : 1.0e300;
      a.partial[(int64_t)tile * 4 + 1] = mass;
      a.partial[(int64_t)tile * 4 + 2] = etot;
      a.partial[(int64_t)tile * 4 + 3] = eint;
    }
  }

  // ---- E. boundary fluxes for the fine-to-coarse correction --------------------
  if (a.tile_corr_off != nullptr) {
    const int n = corr_range[1] - corr_range[0];
    for (int it = tid; it < n * 20; it += NT) {
      const int i = it / 20, r = it % 20;
      const int ent = corr_ent[2 * i], slot = corr_ent[2 * i + 1];
      const int o = ent & 0xff, face = ent >> 8;   // face 0..5 = -x,+x,-y,+y,-z,+z
      const int ox = o % (TX / 2), oy = (o / (TX / 2)) % (TY / 2), oz = o / ((TX / 2) * (TY / 2));
      const int cc = r / 5, v = r % 5;
      const int d = face >> 1, side = face & 1;
      const int t1 = cc & 1, t2 = cc >> 1;
      int fidx;
      if (d == 0) { const int fx = 2 * ox + 2 * side; fidx = fx + (TX + 1) * ((2 * oy + t1) + TY * (2 * oz + t2)); }
      else if (d == 1) { const int fy = 2 * oy + 2 * side; fidx = NFX + (2 * ox + t1) + TX * (fy + (TY + 1) * (2 * oz + t2)); }
      else { const int fz = 2 * oz + 2 * side; fidx = NFX + NFY + (2 * ox + t1) + TX * ((2 * oy + t2) + TY * fz); }
      a.corr_flux[(int64_t)slot * 120 + face * 20 + r] = (double)F.at(fidx, v);
      if (PF && v < 2) a.corr_tmp[(int64_t)slot * 48 + face * 8 + cc * 2 + v] = (double)Ls.at(fidx, v);
    }
  }
}

}  // namespace rb
