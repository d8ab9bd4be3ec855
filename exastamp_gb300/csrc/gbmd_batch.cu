// gbmd_batch.cu -- many independent periodic eam_alloy replicas of uneven
// size in one persistent launch: forward (energy, forces, virial) and the
// parameter adjoint of a force-matching + energy loss.
//
// One thread block owns one replica at a time (replicas are taken largest
// first from an atomic queue, so the launch load-balances uneven sizes), with
// T = 1 .. 32 lanes per atom so that a replica of any size keeps its block's
// threads busy.  Everything a replica needs lives in shared memory: its
// cell-sorted FP32 cell-relative positions with F'(rho), cell ranges, rho, and
// the loss gradients with respect to its per-atom forces and energies.  Pairs
// are found once per replica from the (2S+1)^3 cells around each atom (S = 1
// with cells >= rcut, or S = 2 with cells >= rcut/2), with the same FP32
// screen + FP64 re-test of the ambiguous band as the main path, so the
// in-cutoff pair set is the FP64 one; they go to a pair list in the block's
// own global scratch (at least 2 x 128 entries per atom), which the density,
// force and adjoint passes read, four entries a lane in flight.  A replica with a
// fuller atom walks the cells in every pass instead.  Pair arithmetic is FP32
// with force, energy and density sums compensated pair by pair; per-replica sums
// (energy, virial, loss, gradient) are FP64 and written to the replica's own row.
// Neither depends on which block ran the replica, nor for replicas of up to 512
// atoms on the block's size: their results are the same bit for bit in any batch.
//
// What bounds it: with one lane per atom and one pair in flight, latency (256
// replicas of 243 atoms took 538 us, forward and adjoint, now 192; 4,096 of
// 32-2,048 atoms 11.2 ms, now 4.3).  Of the latter the derivative tables' reads
// (358 KB in use, from L2) are a third, the list a sixth.  The FP64 pipe is slow (16 SM cycles a warp
// instruction), so conversions and the periodic wrap are integer arithmetic,
// the geometry is computed once per replica, and the block sums are
// transposed as they are reduced.
//
// Physics restated (single element, eam_alloy.h L198-313 and
// eam_force_op_multimat.h L114-343):
//   rho_i = sum_j rho(r_ij),  E_i = F(rho_i) + 1/2 sum_j phi(r_ij)
//   f_i   = sum_j u_ij (F'_i rho'(r) + F'_j rho'(r) + phi'(r))
// Adjoint (per parameter theta, derivative splines D of the tables):
//   s_ij = gF_i . u_ij,  G_i = sum_j (s_ij + s_ji) rho'_ij,
//   lam_i = gE_i F'_i + G_i F''_i
//   dL/dtheta = sum_i [gE_i dF + G_i dF'] + sum_ij [ (gE_i/2r - s_ij/r^2) dz2
//               + (s_ij/r) dz2' + s_ij (F'_i + F'_j) drho' + lam_i drho ]
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstring>
#include <numeric>
#include <vector>

#include "gbmd_batch_grid.h"
#include "gbmd_internal.cuh"

namespace {

constexpr int BMAX_ATOMS = 2048;   // largest replica
constexpr int BMAX_CELLS = 1024;
constexpr int SMALL_ATOMS = 512;   // replicas up to this size run in the small-block kernel
constexpr int SMALL_CELLS = 512;
constexpr int NBL_MAX = 256;       // pair-list entries per atom, half of them for either half-warp of the builder
constexpr int BMAX_PARAMS = 9;
constexpr int REP_ROW = 20;  // epot, virial[9], loss, grad[9]
constexpr int MAX_TABLES = 24;  // derivative tables per knot: up to 2 x 9, padded to a multiple of 8

struct BatchArgs {
  int nrep, single;
  const int64_t* off;
  const double* lo;
  const double* hi;
  const double* L;
  const double *x, *y, *z;
  double *fx, *fy, *fz, *ep;
  double* rep;  // nrep x REP_ROW
  const int* order;
  int* queue;
  int* err;
  // tables (FP32 value coefficients c3..c6, scaled by conv)
  const float4 *frho4, *rhor4;
  const float4* fz8;  // per knot: rho' coefficients (3c3, 2c4, c5) / dr, z2r coefficients
  int nr, nrho;
  float rdr, rdrho, rhomax;
  double rcut, rcut2;
  int S;
  // adjoint
  const double *Ftx, *Fty, *Ftz, *Et;
  double wF, wE;
  const float4* dtab;    // [knot][ktab]: derivative tables of z2r (nz2), then of rho (nrh), zero-padded
  const float4* dfrho4;  // [k][knot] for the listed parameters
  int nz2, nrh, nfr, ktab;
  uint32_t* nbl;  // MAXA * NBL_MAX entries per block: the current replica's pair list
  int pz2[BMAX_PARAMS], prh[BMAX_PARAMS], pfr[BMAX_PARAMS];
};

struct RepGeom {
  int64_t base;
  int n, nc[3], ncells, tsh;  // 1 << tsh lanes per atom
  double lo[3], hi[3], L[3], h[3], inv_h[3];
  float hf[3], rc2lo, rc2hi;  // cell edges; FP64 re-test band of the cutoff
};

// One warp's 32 pairs on their way to the derivative tables: knot, and the
// weights of the four coefficients of a z2r and of a rho table.
struct PairRecord {
  float4 z[32], r[32];
  int m[32];
};

// Shared memory of one block: a replica of up to MAXA atoms in MAXC cells.
template <int MAXA, int MAXC, int MAXT>
struct SmemT {
  static constexpr uint32_t ATOMS = MAXA;  // a power of two of at most 2,048
  static constexpr int ROWS = MAXT / 32;
  // replicas that MAXT threads take in one go: every turn of a smaller block has
  // its own rows of red; larger replicas take several goes of the block as it is
  static constexpr bool TURNS = MAXA <= MAXT;
  float4 pos[MAXA];   // by slot: cell-relative FP32 position, w = F'(rho)
  float4 gfe[MAXA];   // adjoint: dL/dF (xyz) and dL/dE (w) by slot; before that, positions by atom
  PairRecord rec[MAXT / 32];
  double red[MAXT / 32][MAX_TABLES];  // block reductions
  RepGeom geom;
  float rho[MAXA];    // by slot: rho, then the adjoint's lambda
  int cfill[MAXC];
  unsigned short cstart[MAXC + 2];
  unsigned short cellof[MAXA];   // by local atom index
  unsigned short order[MAXA];    // slot -> local atom index
  unsigned short nnb[MAXA];      // pair-list length by slot
  unsigned short front[MAXA];    // entries in its first part
  int rep;
  int overflow;             // some atom's pairs do not fit in the list
};

__device__ __forceinline__ int floor_div(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }

// periodic wrap with the rounding of the main path's rebuild (and the oracle)
__device__ __forceinline__ void wrap_cell(const RepGeom& g, double v, int d, double& w, int& c) {
  const long long k = order_key(v);
  if (k <= order_key(g.lo[d]) || k >= order_key(g.hi[d])) {  // outside, or on the face
    if (v < g.lo[d]) v = __dadd_rn(v, g.L[d]);
    else if (v >= g.hi[d]) v = __dsub_rn(v, g.L[d]);
  }
  w = v;
  int q = (int)__dmul_rn(__dsub_rn(v, g.lo[d]), g.inv_h[d]);
  c = q < 0 ? 0 : (q > g.nc[d] - 1 ? g.nc[d] - 1 : q);
}

// Exact FP64 re-test of a pair in the ambiguous band (positions re-read and
// re-wrapped from global memory).
__device__ __noinline__ bool batch_exact(const BatchArgs& A, const RepGeom& g, int ai, int ak, int nx, int ny,
                                         int nz) {
  double wi[3], wk[3];
  int c;
  const double xi[3] = {A.x[g.base + ai], A.y[g.base + ai], A.z[g.base + ai]};
  const double xk[3] = {A.x[g.base + ak], A.y[g.base + ak], A.z[g.base + ak]};
  for (int d = 0; d < 3; ++d) {
    wrap_cell(g, xi[d], d, wi[d], c);
    wrap_cell(g, xk[d], d, wk[d], c);
  }
  double dx, dy, dz;
  return exact_d2(wi[0], wi[1], wi[2], wk[0], wk[1], wk[2], (double)nx * g.L[0], (double)ny * g.L[1],
                  (double)nz * g.L[2], dx, dy, dz) <= A.rcut2;
}

__device__ __forceinline__ float sval(const float4& c, float q) { return fmaf(fmaf(fmaf(c.x, q, c.y), q, c.z), q, c.w); }
__device__ __forceinline__ float sdq(const float4& c, float q) {  // d value / d q
  return fmaf(fmaf(3.f * c.x, q, 2.f * c.y), q, c.z);
}

// Embedding knot of rho, and the fraction (linear continuation above the table
// is the caller's).
__device__ __forceinline__ int embed_knot(const BatchArgs& A, float rho, float& q) {
  q = fmaf(rho, A.rdrho, 1.f);
  const int m = max(1, min((int)q, A.nrho - 1));
  q = fminf(q - (float)m, 1.f);
  return m;
}

__device__ __forceinline__ int knot(float t, int nmax, float& q) {
  const int m = min((int)t, nmax);
  q = fminf(t - (float)m, 1.0f);
  return m;
}

// FP32 separation of a candidate (position shifted by its cell offset) and
// its square: the one expression every pass and the list build use.
__device__ __forceinline__ float pair_d2(const float4& pi, const float4& pj, float sx, float sy, float sz,
                                         float& ddx, float& ddy, float& ddz) {
  ddx = (pj.x - pi.x) + sx;
  ddy = (pj.y - pi.y) + sy;
  ddz = (pj.z - pi.z) + sz;
  return fmaf(ddx, ddx, fmaf(ddy, ddy, ddz * ddz));
}

// Lane t of atom s's T lanes: every T-th candidate of each cell around slot s,
// fn(k, dx, dy, dz, d2, code) where it lies within the cutoff, code = the cell
// offset (dx+S) | (dy+S) << 3 | (dz+S) << 6.
template <class SM, class Fn>
__device__ __forceinline__ void for_pairs(const BatchArgs& A, const RepGeom& g, const SM& sm, int s, int t, int T,
                                          Fn fn) {
  const int ai = sm.order[s];
  const int c = sm.cellof[ai];
  const int cx = c % g.nc[0], cy = (c / g.nc[0]) % g.nc[1], cz = c / (g.nc[0] * g.nc[1]);
  const float4 pi = sm.pos[s];
  const int S = A.S;
  for (int dz = -S; dz <= S; ++dz) {
    const int vz = cz + dz, nz = floor_div(vz, g.nc[2]), wz = vz - nz * g.nc[2];
    for (int dy = -S; dy <= S; ++dy) {
      const int vy = cy + dy, ny = floor_div(vy, g.nc[1]), wy = vy - ny * g.nc[1];
      for (int dx = -S; dx <= S; ++dx) {
        const int vx = cx + dx, nx = floor_div(vx, g.nc[0]), wx = vx - nx * g.nc[0];
        const int cj = (wz * g.nc[1] + wy) * g.nc[0] + wx;
        const float sx = (float)dx * g.hf[0], sy = (float)dy * g.hf[1], sz = (float)dz * g.hf[2];
        const bool self_cell = (dx | dy | dz) == 0;
        const uint32_t code = (uint32_t)(dx + S) | ((uint32_t)(dy + S) << 3) | ((uint32_t)(dz + S) << 6);
        for (int k = sm.cstart[cj] + t; k < sm.cstart[cj + 1]; k += T) {
          if (self_cell && k == s) continue;
          float ddx, ddy, ddz;
          const float d2 = pair_d2(pi, sm.pos[k], sx, sy, sz, ddx, ddy, ddz);
          if (!(d2 <= g.rc2hi) || (d2 >= g.rc2lo && !batch_exact(A, g, ai, sm.order[k], nx, ny, nz))) continue;
          fn(k, ddx, ddy, ddz, d2, code);
        }
      }
    }
  }
}

// The pair list of a replica of n atoms: entries (slot k | code << 11) in two
// parts per atom of up to cap entries, entry q of part p of slot s in word
// (p cap + q) n + s; the first `front` entries of the atom are its part 0, the
// rest part 1.  Read past L1, which serves the tables.
struct PairList {
  const uint32_t* at;
  int front, count, n, jump;
  template <class SM>
  __device__ __forceinline__ PairList(const SM& sm, const uint32_t* nbl, int n_, int cap, int s)
      : at(nbl + s), front(min((int)sm.front[s], cap)), count(min((int)sm.nnb[s], front + cap)), n(n_), jump(cap - front) {}
  __device__ __forceinline__ uint32_t operator[](int e) const {
    uint32_t w;
    asm volatile("ld.global.L1::no_allocate.u32 %0, [%1];" : "=r"(w) : "l"(at + (e < front ? e : e + jump) * n));
    return w;
  }
};

// {0 .. 2S} -> -S .. S exactly (small integer through the 2^23 mantissa trick)
__device__ __forceinline__ float cell_unit(uint32_t b, float bias) { return __int_as_float(0x4B000000u | b) - bias; }

// Lane t's share of the pairs of slot s, fn(k, dx, dy, dz, d2, ok), four at a
// time; pairs with ok = false count nothing (their separation is zero).  From the list, or from the cells (cap = 0) where some
// atom's pairs do not fit in it.
template <class SM, class Fn>
__device__ __forceinline__ void visit(const BatchArgs& A, const RepGeom& g, const SM& sm, const uint32_t* nbl,
                                      int cap, int s, int t, Fn fn) {
  const int T = 1 << g.tsh;
  if (cap == 0) {
    for_pairs(A, g, sm, s, t, T, [&](int k, float dx, float dy, float dz, float d2, uint32_t) {
      fn(k, dx, dy, dz, d2, true);
    });
    return;
  }
  const float4 pi = sm.pos[s];
  const PairList list(sm, nbl, g.n, cap, s);
  const float bias = 8388608.0f + (float)A.S;
  const uint32_t none = (uint32_t)s | (uint32_t)(A.S | (A.S << 3) | (A.S << 6)) << 11;
  const int n = list.count;
  uint32_t e[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) e[u] = t + u * T < n ? list[t + u * T] : none;
  for (int q = t; q < n; q += 4 * T) {
    uint32_t nxt[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) nxt[u] = q + (4 + u) * T < n ? list[q + (4 + u) * T] : none;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = (int)(e[u] & (SM::ATOMS - 1u));
      const float sx = cell_unit((e[u] >> 11) & 7u, bias) * g.hf[0], sy = cell_unit((e[u] >> 14) & 7u, bias) * g.hf[1],
                  sz = cell_unit((e[u] >> 17) & 7u, bias) * g.hf[2];
      float ddx, ddy, ddz;
      const float d2 = pair_d2(pi, sm.pos[k], sx, sy, sz, ddx, ddy, ddz);
      fn(k, ddx, ddy, ddz, d2, q + u * T < n);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) e[u] = nxt[u];
  }
}

// The replica's pair list, by warps: a warp takes 16 atoms of a cell, lanes l
// and l + 16 hold atom l.  The candidates of up to 32 stencil cells at a time
// are staged in shared memory, 32 for each half-warp, without those farther
// than the cutoff from the group's bounding box; the low half-warp tests the
// first half of them and writes its hits to part 0 of the atom's list, the high
// one tests the second half and writes part 1.  The walk of the main path's
// list builder, with the rows in the block's scratch (L2) instead of shared
// memory.  A test costs some ten instructions of a warp; one lane walking the
// cells of its own atom took 45, half of the whole evaluation (243 atoms:
// 200,000 of 420,000 cycles).  A part of more than cap - 4 entries raises
// sm.overflow, and the passes walk the cells.
template <int MAXT, class SM>
__device__ void build_list(const BatchArgs& A, const RepGeom& g, SM& sm, uint32_t* __restrict__ nbl, int cap) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int half = lane >> 4, hl = lane & 15, S = A.S, width = 2 * S + 1, ncells = width * width * width;
  const int n = g.n;
  // staging: x, y, z, entry of the low half's 32 candidates, then the high
  // half's, 64 bytes further (other banks); the cells' shifts, x = (first slot
  // - first candidate) << 9 | code
  float* const chunk = reinterpret_cast<float*>(&sm.rec[wid]);
  float4* const shift = sm.gfe + 32 * wid;
  static_assert(sizeof(PairRecord) >= (2 * 128 + 16) * sizeof(float), "staging fits");
  int item = wid;  // groups of 16 atoms, cell by cell, dealt to the warps in turn
  for (int cell = 0; cell < g.ncells; ++cell) {
    const int b = sm.cstart[cell], nh = sm.cstart[cell + 1] - b;
    for (int h0 = 0; h0 < nh; h0 += 16, --item) {
      if (item != 0) continue;
      item = nw;
      const bool hv = h0 + hl < nh;
      const int s = b + h0 + hl;
      const float FAR = 1e18f;
      float4 pi = make_float4(FAR, FAR, FAR, 0.f);
      if (hv) pi = sm.pos[s];
      float3 blo = make_float3(pi.x, pi.y, pi.z);
      float3 bhi = make_float3(hv ? pi.x : -FAR, hv ? pi.y : -FAR, hv ? pi.z : -FAR);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        blo.x = fminf(blo.x, __shfl_xor_sync(FULL, blo.x, o));
        blo.y = fminf(blo.y, __shfl_xor_sync(FULL, blo.y, o));
        blo.z = fminf(blo.z, __shfl_xor_sync(FULL, blo.z, o));
        bhi.x = fmaxf(bhi.x, __shfl_xor_sync(FULL, bhi.x, o));
        bhi.y = fmaxf(bhi.y, __shfl_xor_sync(FULL, bhi.y, o));
        bhi.z = fmaxf(bhi.z, __shfl_xor_sync(FULL, bhi.z, o));
      }
      const float keep2 = g.rc2hi * (1.0f + 0x1p-10f);  // far above the rounding of the tests' d2
      const float2 npx = make_float2(-pi.x, -pi.x), npy = make_float2(-pi.y, -pi.y), npz = make_float2(-pi.z, -pi.z);
      const uint32_t self = (uint32_t)s | (uint32_t)(S | (S << 3) | (S << 6)) << 11;
      const int cx = cell % g.nc[0], cy = (cell / g.nc[0]) % g.nc[1], cz = cell / (g.nc[0] * g.nc[1]);
      uint32_t* const part = nbl + (size_t)half * cap * n + s;  // this lane's: entry q at part[q n]
      uint32_t* put = part;
      const uint32_t* const last = part + (size_t)(cap - 4) * n;
      const long long step = 4ll * n;
      int cnt = 0;
      float thr = hv ? g.rc2hi : -1.f;  // -1: no candidate is a hit
      float far2 = -1.f;                // largest d2 of the hits
      for (int c0 = 0; c0 < ncells; c0 += 32) {
        // stencil cell of this lane
        int start = 0, many = 0;
        float4 sh = make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t code = 0;
        if (c0 + lane < ncells) {
          const int q = c0 + lane, dx = q % width - S, dy = (q / width) % width - S, dz = q / (width * width) - S;
          const int vx = cx + dx, vy = cy + dy, vz = cz + dz;
          const int wx = vx - floor_div(vx, g.nc[0]) * g.nc[0], wy = vy - floor_div(vy, g.nc[1]) * g.nc[1],
                    wz = vz - floor_div(vz, g.nc[2]) * g.nc[2];
          const int cj = (wz * g.nc[1] + wy) * g.nc[0] + wx;
          start = sm.cstart[cj];
          many = sm.cstart[cj + 1] - start;
          sh = make_float4(0.f, (float)dx * g.hf[0], (float)dy * g.hf[1], (float)dz * g.hf[2]);
          code = (uint32_t)(dx + S) | ((uint32_t)(dy + S) << 3) | ((uint32_t)(dz + S) << 6);
        }
        int incl = many;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(FULL, incl, o);
          if (lane >= o) incl += v;
        }
        const int pre = incl - many, total = __shfl_sync(FULL, incl, 31);
        const bool any = many > 0;
        const unsigned anyb = __ballot_sync(FULL, any);
        __syncwarp();
        if (any) {
          sh.x = __int_as_float(((start - pre) << 9) | (int)code);
          shift[__popc(anyb & ((1u << lane) - 1u))] = sh;
        }
        const int mid = min(total, (((total + 1) >> 1) + 31) & ~31);
        for (int qa = 0; qa < mid; qa += 32) {
          __syncwarp();
          int m[2];
#pragma unroll
          for (int side = 0; side < 2; ++side) {
            const int w0 = side ? total - qa - 32 : qa, q0 = side ? mid : 0, q1 = side ? total : mid;
            const int off = pre - w0, q = w0 + lane;
            const unsigned starts = __reduce_or_sync(FULL, any && (unsigned)off < 32u ? 1u << off : 0u);
            const int before = __popc(__ballot_sync(FULL, any && off < 0));
            const bool valid = q >= q0 && q < q1;
            const int sc = valid ? before + __popc(starts & (0xffffffffu >> (31 - lane))) - 1 : 0;
            const float4 cs = shift[sc];
            const int dc = __float_as_int(cs.x), k = valid ? q + (dc >> 9) : 0;
            const float4 pj = sm.pos[k];
            // the separation's rounding is pair_d2's, (p_j - p_i) + shift, below;
            // here the shifted position serves the box test alone
            const float ex = pj.x + cs.y, ey = pj.y + cs.z, ez = pj.z + cs.w;
            const float bx = fmaxf(0.f, fmaxf(blo.x - ex, ex - bhi.x));
            const float by = fmaxf(0.f, fmaxf(blo.y - ey, ey - bhi.y));
            const float bz = fmaxf(0.f, fmaxf(blo.z - ez, ez - bhi.z));
            const bool keep = valid && fmaf(bx, bx, fmaf(by, by, bz * bz)) <= keep2;
            const unsigned km = __ballot_sync(FULL, keep), lt = (1u << lane) - 1u;
            m[side] = __popc(km);
            float* const d = chunk + side * (128 + 16) + (keep ? __popc(km & lt) : m[side] + __popc(~km & lt));
            d[0] = keep ? ex : FAR;
            d[32] = ey;
            d[64] = ez;
            d[96] = __uint_as_float((uint32_t)k | (uint32_t)(dc & 511) << 11);
          }
          __syncwarp();
          const int mm = max(m[0], m[1]);
          const float4* const cand = reinterpret_cast<const float4*>(chunk + half * (128 + 16));
          for (int t = 0; t < mm; t += 4) {
            if (put > last) {
              thr = -1.f;
              sm.overflow = 1;
            }
            const float4 x = cand[t / 4], y = cand[8 + t / 4], z = cand[16 + t / 4], w = cand[24 + t / 4];
            const float2 dx0 = __fadd2_rn(make_float2(x.x, x.y), npx), dx1 = __fadd2_rn(make_float2(x.z, x.w), npx);
            const float2 dy0 = __fadd2_rn(make_float2(y.x, y.y), npy), dy1 = __fadd2_rn(make_float2(y.z, y.w), npy);
            const float2 dz0 = __fadd2_rn(make_float2(z.x, z.y), npz), dz1 = __fadd2_rn(make_float2(z.z, z.w), npz);
            const float2 d0 = __ffma2_rn(dx0, dx0, __ffma2_rn(dy0, dy0, __fmul2_rn(dz0, dz0)));
            const float2 d1 = __ffma2_rn(dx1, dx1, __ffma2_rn(dy1, dy1, __fmul2_rn(dz1, dz1)));
            const float dd[4] = {d0.x, d0.y, d1.x, d1.y};
            const uint32_t ww[4] = {__float_as_uint(w.x), __float_as_uint(w.y), __float_as_uint(w.z),
                                    __float_as_uint(w.w)};
#pragma unroll
            for (int u = 0; u < 4; ++u)  // predicated: four tests are one straight line
              asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 q, %5, %7;\nsetp.le.and.f32 p, %3, %4, q;\n"
                           "@p st.global.u32 [%0], %5;\n@p add.s64 %0, %0, %6;\n@p add.s32 %1, %1, 1;\n"
                           "@p max.f32 %2, %2, %3;\n}"
                           : "+l"(put), "+r"(cnt), "+f"(far2)
                           : "f"(dd[u]), "f"(thr), "r"(ww[u]), "l"(step), "r"(self)
                           : "memory");
          }
        }
      }
      // exact re-test of the band entries, by the lane that wrote them
      int kept = cnt;
      if (hv && far2 >= g.rc2lo * (1.0f - 0x1p-20f)) {
        int to = 0;
        for (int q = 0; q < cnt; ++q) {
          const uint32_t w = part[(size_t)q * n];
          const int k = (int)(w & 2047u), dx = (int)((w >> 11) & 7u) - S, dy = (int)((w >> 14) & 7u) - S,
                    dz = (int)(w >> 17) - S;
          float ddx, ddy, ddz;
          const float d2 = pair_d2(pi, sm.pos[k], (float)dx * g.hf[0], (float)dy * g.hf[1], (float)dz * g.hf[2], ddx,
                                   ddy, ddz);
          if (d2 < g.rc2lo || (d2 <= g.rc2hi && batch_exact(A, g, sm.order[s], sm.order[k], floor_div(cx + dx, g.nc[0]),
                                                            floor_div(cy + dy, g.nc[1]), floor_div(cz + dz, g.nc[2]))))
            part[(size_t)(to++) * n] = w;
        }
        kept = to;
      }
      const int other = __shfl_xor_sync(FULL, kept, 16);
      if (hv && half == 0) {
        sm.front[s] = (unsigned short)kept;
        sm.nnb[s] = (unsigned short)(kept + other);
      }
    }
  }
}

// Merge the compensated sums of an atom's T lanes (all lanes of the warp).
__device__ __forceinline__ void reduce_kahan(float& s, float& c, int T) {
  for (int off = T >> 1; off > 0; off >>= 1) {
    const float s2 = __shfl_xor_sync(0xffffffffu, s, off), c2 = __shfl_xor_sync(0xffffffffu, c, off);
    kahan_merge(s, c, s2, c2);
  }
}
__device__ __forceinline__ void reduce_plain(float& s, int T) {
  for (int off = T >> 1; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
}

__device__ __forceinline__ void knot_pair(const float4* p, float4& a, float4& b) {
  asm("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(p));
}

// Block barrier after code in which lanes of a warp part (a last warp with
// fewer atoms than lanes, lists of different lengths): the warp comes together
// first.  With one lane per atom nothing else brings the lanes of a short warp
// together before the barrier, and it was seen to count such a warp twice.
__device__ __forceinline__ void block_sync() {
  __syncwarp();
  __syncthreads();
}

// The block's sums of NV quantities, in two steps: a warp's to row `row` of red,
// and the first `rows` rows' to red[0][0 .. NV).  The atoms are dealt out over
// MAXT threads whatever the block has: a block of fewer takes them in several
// turns, and each turn of each of its warps has a row of its own, so that a
// replica's sums are added in one order whatever the block (SmemT::turn_row).
template <int NV, class SM>
__device__ __forceinline__ void warp_sums(SM& sm, double (&v)[NV], int row) {
  const int q = warp_sum_transposed<NV>(v, threadIdx.x & 31);
  if (q >= 0 && row < SM::ROWS) sm.red[row][q] = v[0];
}

template <int NV, class SM>
__device__ __forceinline__ void block_sums(SM& sm, int rows) {
  block_sync();
  if (threadIdx.x < NV) {
    double a = 0.0;
    for (int k = 0; k < rows; ++k) a += sm.red[k][threadIdx.x];
    sm.red[0][threadIdx.x] = a;
  }
  block_sync();
}

template <int MAXA, int MAXC, int MAXT, int MINB, bool ADJ>
__global__ void __launch_bounds__(MAXT, MINB) k_batch(const __grid_constant__ BatchArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using SM = SmemT<MAXA, MAXC, MAXT>;
  SM& sm = *reinterpret_cast<SM*>(smem_raw);
  const int tid = threadIdx.x, B = blockDim.x;
  RepGeom& g = sm.geom;
  // Persistent mode: take queue tickets until they run past nrep (each block
  // takes at most nrep + 1 tickets).  Single mode: exactly one replica.
  for (int iter = 0;; ++iter) {
    if (tid == 0) sm.rep = A.single >= 0 ? (iter == 0 ? A.single : A.nrep) : atomicAdd(A.queue, 1);
    block_sync();
    const int qi = sm.rep;
    if (qi < 0 || qi >= A.nrep) break;
    const int r = A.single >= 0 ? qi : A.order[qi];
    double* row = A.rep + (size_t)r * REP_ROW;
    for (int c = tid; c < MAXC; c += B) sm.cfill[c] = 0;
    if (tid < 3) {  // FP64 divisions take some 600 cycles each: few of them in a row
      const int d = tid;
      const double L3[3] = {A.L[3 * r], A.L[3 * r + 1], A.L[3 * r + 2]};
      int nc[3];
      const int ncells = gbmd::batch_grid_dims(L3, A.rcut, A.S, MAXC, nc);
      const double L = L3[d];
      const double n = small_double(d == 0 ? nc[0] : (d == 1 ? nc[1] : nc[2]));
      g.lo[d] = A.lo[3 * r + d];
      g.hi[d] = A.hi[3 * r + d];
      g.L[d] = L;
      g.nc[d] = (int)n;
      g.h[d] = L / n;
      g.inv_h[d] = n / L;
      g.hf[d] = (float)g.h[d];
      if (d == 0) {
        g.base = A.off[r];
        g.n = (int)(A.off[r + 1] - g.base);
        g.ncells = ncells;
        int tsh = 0;  // the most lanes per atom with which MAXT threads take the replica in one go
        while (tsh < 5 && (g.n << (tsh + 1)) <= (SM::TURNS ? MAXT : B)) ++tsh;
        g.tsh = tsh;
        sm.overflow = 0;
        // the band covers the rounding of coordinates in cells of edge h, as
        // band_tol's does for its cells
        const float hmax = fmaxf((float)L3[0] / nc[0], fmaxf((float)L3[1] / nc[1], (float)L3[2] / nc[2]));
        const float rc = (float)A.rcut, band = fminf(0x1p-16f * fmaxf(1.f, hmax / rc), 0.5f);
        g.rc2lo = rc * rc * (1.f - band);
        g.rc2hi = rc * rc * (1.f + band);
      }
    }
    block_sync();
    const int n = g.n;
    if (n > MAXA || g.L[0] < A.rcut || g.L[1] < A.rcut || g.L[2] < A.rcut) {
      if (tid == 0) {
        atomicOr(&A.err[0], 16);
        for (int q = 0; q < REP_ROW; ++q) row[q] = __longlong_as_double(0x7ff8000000000000ll);
      }
      block_sync();
      continue;
    }
    // ---- cell sort (deterministic order inside a cell: local atom index)
    for (int a = tid; a < n; a += B) {
      const double xs[3] = {A.x[g.base + a], A.y[g.base + a], A.z[g.base + a]};
      int c3[3];
      float lp[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        double w;
        wrap_cell(g, xs[d], d, w, c3[d]);
        lp[d] = narrow(w - small_double(c3[d]) * g.h[d] - g.lo[d]);
      }
      const int c = (c3[2] * g.nc[1] + c3[1]) * g.nc[0] + c3[0];
      sm.cellof[a] = (unsigned short)c;
      sm.gfe[a] = make_float4(lp[0], lp[1], lp[2], 0.f);
      atomicAdd(&sm.cfill[c], 1);
    }
    block_sync();
    if (tid < 32) {  // warp scan of the cell counts
      const int per = (g.ncells + 31) / 32;
      int loc = 0;
      for (int k = 0; k < per; ++k) {
        const int c = tid * per + k;
        if (c < g.ncells) loc += sm.cfill[c];
      }
      int inc = loc;
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (tid >= o) inc += v;
      }
      int run = inc - loc;
      for (int k = 0; k < per; ++k) {
        const int c = tid * per + k;
        if (c < g.ncells) {
          sm.cstart[c] = (unsigned short)run;
          run += sm.cfill[c];
          sm.cfill[c] = 0;
        }
      }
      if (tid == 31) sm.cstart[g.ncells] = (unsigned short)inc;
    }
    block_sync();
    for (int a = tid; a < n; a += B) {  // any order first
      const int c = sm.cellof[a];
      sm.nnb[sm.cstart[c] + atomicAdd(&sm.cfill[c], 1)] = (unsigned short)a;
    }
    block_sync();
    for (int s = tid; s < n; s += B) {  // then by rank among the cell's atoms
      const int a = sm.nnb[s], c = sm.cellof[a], b = sm.cstart[c], e = sm.cstart[c + 1];
      int rank = b;
      for (int k = b; k < e; ++k) rank += sm.nnb[k] < a;
      sm.order[rank] = (unsigned short)a;
      sm.pos[rank] = sm.gfe[a];
    }
    block_sync();
    const int T = 1 << g.tsh, t = tid & (T - 1), ns = B >> g.tsh;  // ns atoms at a time
    const int rows = SM::TURNS ? ((n << g.tsh) + 31) >> 5 : B >> 5;  // of red that hold sums
    // ---- pair list: one walk over the cells (FP32 screen, FP64 band
    // re-test), then every pass below reads the list
    uint32_t* nbl = A.nbl + (A.single >= 0 ? (size_t)0 : (size_t)blockIdx.x * MAXA * NBL_MAX);
    const int cap = MAXA * NBL_MAX / (2 * max(n, 1));  // entries in either part
    build_list<MAXT>(A, g, sm, nbl, cap);
    block_sync();
    const bool list_ok = !sm.overflow;
    const int listed = list_ok ? cap : 0;
    // ---- density + embedding
    for (int s0 = 0; s0 < n; s0 += ns) {
      const int s = s0 + (tid >> g.tsh);
      float acc = 0.f, comp = 0.f;
      if (s < n)
        visit(A, g, sm, nbl, listed, s, t,
              [&](int k, float dx, float dy, float dz, float d2, bool ok) {
                const float rr = d2 * rsqrtf(d2);
                float q;
                const int m = knot(fmaf(rr, A.rdr, 1.f), A.nr - 1, q);
                const float val = sval(A.rhor4[m], q);
                kahan_add(acc, comp, ok ? val : 0.f);
              });
      reduce_kahan(acc, comp, T);
      if (s < n && t == 0) sm.rho[s] = acc - comp;
    }
    block_sync();
    // F'(rho); E = F(rho) is formed again where it is needed
    for (int s = tid; s < n; s += B) {
      float q;
      const float4 c = A.frho4[embed_knot(A, sm.rho[s], q)];
      sm.pos[s].w = sdq(c, q) * A.rdrho;
    }
    block_sync();
    // ---- forces, energies, virial; loss residuals
    // block sums: energy, virial xx yy zz xy xz yz, loss
    constexpr int NV = ADJ ? 8 : 7;
    double sum[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) sum[q] = 0.0;
    int row_of = tid >> 5;
    for (int s0 = 0; s0 < n; s0 += ns) {
      const int s = s0 + (tid >> g.tsh);
      float fx = 0.f, fy = 0.f, fz = 0.f, cx = 0.f, cy = 0.f, cz = 0.f, ee = 0.f, ce = 0.f;
      float v[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (s < n) {
        const float fpi = sm.pos[s].w;
        visit(A, g, sm, nbl, listed, s, t,
              [&](int k, float dx, float dy, float dz, float d2, bool ok) {
                const float rs = rsqrtf(d2), rr = d2 * rs;
                float q;
                const int m = knot(fmaf(rr, A.rdr, 1.f), A.nr - 1, q);
                float4 dr, cz2;
                knot_pair(A.fz8 + 2 * m, dr, cz2);
                const float rhop = fmaf(fmaf(dr.x, q, dr.y), q, dr.z);
                const float z2 = sval(cz2, q), z2d = sdq(cz2, q) * A.rdr;
                const float phi = z2 * rs;
                const float phip = (z2d - phi) * rs;
                const float psip = fmaf(fpi + sm.pos[k].w, rhop, phip);
                const float fpair = ok ? psip * rs : 0.f;
                kahan_add(fx, cx, dx * fpair);
                kahan_add(fy, cy, dy * fpair);
                kahan_add(fz, cz, dz * fpair);
                kahan_add(ee, ce, ok ? 0.5f * phi : 0.f);
                const float hh = -0.5f * fpair;
                v[0] = fmaf(hh * dx, dx, v[0]);
                v[1] = fmaf(hh * dy, dy, v[1]);
                v[2] = fmaf(hh * dz, dz, v[2]);
                v[3] = fmaf(hh * dx, dy, v[3]);
                v[4] = fmaf(hh * dx, dz, v[4]);
                v[5] = fmaf(hh * dy, dz, v[5]);
              });
      }
      reduce_kahan(fx, cx, T);
      reduce_kahan(fy, cy, T);
      reduce_kahan(fz, cz, T);
      reduce_kahan(ee, ce, T);
#pragma unroll
      for (int q = 0; q < 6; ++q) reduce_plain(v[q], T);
      if (s < n && t == 0) {
        const int64_t ga = g.base + sm.order[s];
        const double Fx = widen(fx - cx), Fy = widen(fy - cy), Fz = widen(fz - cz);
        const float R = sm.rho[s];
        float q;
        const float4 c = A.frho4[embed_knot(A, R, q)];
        float emb = sval(c, q);
        if (R > A.rhomax) emb = fmaf(sm.pos[s].w, R - A.rhomax, emb);
        const double E = widen(emb) + widen(ee - ce);
        A.fx[ga] = Fx;
        A.fy[ga] = Fy;
        A.fz[ga] = Fz;
        A.ep[ga] = E;
        sum[0] += E;
#pragma unroll
        for (int u = 0; u < 6; ++u) sum[1 + u] += widen(v[u]);
        if (ADJ) {
          const double ex = Fx - A.Ftx[ga], ey = Fy - A.Fty[ga], ez = Fz - A.Ftz[ga], de = E - A.Et[ga];
          sum[ADJ ? 7 : 0] += A.wF * (ex * ex + ey * ey + ez * ez) + A.wE * de * de;
          const double twF = 2.0 * A.wF;
          sm.gfe[s] = make_float4(narrow(twF * ex), narrow(twF * ey), narrow(twF * ez), narrow(2.0 * A.wE * de));
        }
      }
      if (SM::TURNS || s0 + ns >= n) {
        __syncwarp();
        warp_sums<NV>(sm, sum, row_of);
        row_of += B >> 5;
#pragma unroll
        for (int q = 0; q < NV; ++q) sum[q] = 0.0;
      }
    }
    block_sums<NV>(sm, rows);
    if (tid < (ADJ ? 11 : 10)) {
      // row-major virial from xx yy zz xy xz yz
      const int q = tid == 0 ? 0 : (tid == 10 ? 7 : 1 + (int)((0x254513430ll >> (4 * (tid - 1))) & 15));
      row[tid] = sm.red[0][q];
    }
    if (!ADJ && tid >= 10 && tid < REP_ROW) row[tid] = 0.0;
    if constexpr (ADJ) {
      double fr[BMAX_PARAMS];  // dF/dtheta terms
#pragma unroll
      for (int p = 0; p < BMAX_PARAMS; ++p) fr[p] = 0.0;
      block_sync();  // red is read
      row_of = tid >> 5;
      // ---- adjoint sweep 1: G_i, then the embedding terms and lambda_i
      for (int s0 = 0; s0 < n; s0 += ns) {
        const int s = s0 + (tid >> g.tsh);
        float Gs = 0.f;
        float4 gi = make_float4(0.f, 0.f, 0.f, 0.f);
        if (s < n) {
          gi = sm.gfe[s];
          visit(A, g, sm, nbl, listed, s, t,
                [&](int k, float dx, float dy, float dz, float d2, bool ok) {
                  const float rs = rsqrtf(d2), rr = d2 * rs;
                  float q;
                  const int m = knot(fmaf(rr, A.rdr, 1.f), A.nr - 1, q);
                  const float ux = dx * rs, uy = dy * rs, uz = dz * rs;
                  const float4 gk = sm.gfe[k];
                  const float sij = fmaf(gi.x, ux, fmaf(gi.y, uy, gi.z * uz));
                  const float sji = -fmaf(gk.x, ux, fmaf(gk.y, uy, gk.z * uz));
                  const float4 dr = A.fz8[2 * m];
                  const float rhop = fmaf(fmaf(dr.x, q, dr.y), q, dr.z);
                  Gs = ok ? fmaf(sij + sji, rhop, Gs) : Gs;
                });
        }
        reduce_plain(Gs, T);
        if (s < n && t == 0) {
          const float R = sm.rho[s];
          float q;
          const int m = embed_knot(A, R, q);
          const float4 c = A.frho4[m];
          const bool over = R > A.rhomax;
          const float f2 = over ? 0.f : fmaf(6.f * c.x, q, 2.f * c.y) * A.rdrho * A.rdrho;
          sm.rho[s] = fmaf(gi.w, sm.pos[s].w, Gs * f2);
#pragma unroll
          for (int p = 0; p < BMAX_PARAMS; ++p)
            if (p < A.nfr) {
              const float4 dc = A.dfrho4[(size_t)p * (A.nrho + 1) + m];
              const float dfp = sdq(dc, q) * A.rdrho;
              fr[p] += widen(fmaf(gi.w, sval(dc, q) + (over ? dfp * (R - A.rhomax) : 0.f), Gs * dfp));
            }
        }
        if (SM::TURNS || s0 + ns >= n) {
          __syncwarp();
          warp_sums<BMAX_PARAMS>(sm, fr, row_of);
          row_of += B >> 5;
#pragma unroll
          for (int p = 0; p < BMAX_PARAMS; ++p) fr[p] = 0.0;
        }
      }
      block_sums<BMAX_PARAMS>(sm, rows);
      if (tid < BMAX_PARAMS) {
        double v = 0.0;
        for (int p = 0; p < A.nfr; ++p)
          if (A.pfr[p] == tid) v += sm.red[0][p];
        row[11 + tid] = v;
      }
      // ---- adjoint sweep 2: the tables' terms.  A pair's contribution to the
      // gradient of any z2r (rho) parameter is the same four weights times its
      // table's four coefficients at the pair's knot.  A lane forms the weights
      // of its pair; then eight lanes take the tables of one pair, 16 bytes of
      // one or a few 128-byte lines each (a lane reading all tables of its own
      // pair costs 32 lines a read).
      const int lane = tid & 31, wid = tid >> 5;
      PairRecord& rec = sm.rec[wid];
      const int nb = A.ktab >> 3;  // table batches of eight
      float acc[MAX_TABLES / 8];
      double accd[MAX_TABLES / 8];
#pragma unroll
      for (int b = 0; b < MAX_TABLES / 8; ++b) {
        acc[b] = 0.f;
        accd[b] = 0.0;
      }
      auto weights = [&](const float4& gi, float fpi, float lam, int k, float dx, float dy, float dz, float d2, bool ok) {
        const float rs = rsqrtf(d2), rr = d2 * rs;
        float q;
        const int m = knot(fmaf(rr, A.rdr, 1.f), A.nr - 1, q);
        const float sij = fmaf(gi.x, dx, fmaf(gi.y, dy, gi.z * dz)) * rs;
        const float wv = (0.5f * gi.w - sij * rs) * rs;        // weight of dz2
        const float wd = sij * rs * A.rdr;                     // of d(dz2)/dq
        const float wr = sij * (fpi + sm.pos[k].w) * A.rdr;    // of d(drho)/dq; lam: of drho
        rec.m[lane] = ok ? m : 0;
        rec.z[lane] = ok ? make_float4(fmaf(wv, q, 3.f * wd) * q * q, fmaf(wv, q, 2.f * wd) * q, fmaf(wv, q, wd), wv)
                         : make_float4(0.f, 0.f, 0.f, 0.f);
        rec.r[lane] = ok ? make_float4(fmaf(lam, q, 3.f * wr) * q * q, fmaf(lam, q, 2.f * wr) * q, fmaf(lam, q, wr), lam)
                         : make_float4(0.f, 0.f, 0.f, 0.f);
      };
      auto tables = [&]() {  // the warp's 32 recorded pairs
        __syncwarp();
        const int kt = lane & 7;
        for (int b = 0; b < nb; ++b) {
          const float4* const w = kt + 8 * b < A.nz2 ? rec.z : rec.r;
          float a = 0.f;
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int pr = 4 * u + (lane >> 3);
            const float4 c = A.dtab[(size_t)rec.m[pr] * A.ktab + kt + 8 * b], f = w[pr];
            a = fmaf(c.x, f.x, fmaf(c.y, f.y, fmaf(c.z, f.z, fmaf(c.w, f.w, a))));
          }
#pragma unroll
          for (int bb = 0; bb < MAX_TABLES / 8; ++bb)
            if (bb == b) acc[bb] += a;
        }
        __syncwarp();
      };
      auto settle = [&]() {
#pragma unroll
        for (int b = 0; b < MAX_TABLES / 8; ++b)
          if (b < nb) {
            accd[b] += widen(acc[b]);
            acc[b] = 0.f;
          }
      };
      // a turn's sums of eight tables at a time, to its row of red
      auto store_tables = [&]() {
#pragma unroll
        for (int b = 0; b < MAX_TABLES / 8; ++b) {
          accd[b] += __shfl_xor_sync(0xffffffffu, accd[b], 8);
          accd[b] += __shfl_xor_sync(0xffffffffu, accd[b], 16);
          if (lane < 8 && row_of < SM::ROWS) sm.red[row_of][lane + 8 * b] = accd[b];
          accd[b] = 0.0;
        }
        row_of += B >> 5;
      };
      block_sync();  // lambda is complete; red is read
      row_of = wid;
      if (nb > 0) {
        const float bias = 8388608.0f + (float)A.S;
        const uint32_t none = (uint32_t)(A.S | (A.S << 3) | (A.S << 6)) << 11;
        for (int s0 = 0; s0 < n && list_ok; s0 += ns) {
          const bool live = s0 + (tid >> g.tsh) < n;
          const int s = live ? s0 + (tid >> g.tsh) : n - 1;
          const float4 gi = sm.gfe[s], pi = sm.pos[s];
          const float lam = sm.rho[s];
          const PairList list(sm, nbl, n, cap, s);
          const int mine = live ? list.count : 0;
          const int steps = __reduce_max_sync(0xffffffffu, mine);
          uint32_t e = t < mine ? list[t] : none | s;
          for (int q = t; q - t < steps; q += T) {
            const uint32_t nxt = q + T < mine ? list[q + T] : none | s;
            const int k = (int)(e & (SM::ATOMS - 1u));
            float dx, dy, dz;
            const float d2 = pair_d2(pi, sm.pos[k], cell_unit((e >> 11) & 7u, bias) * g.hf[0],
                                     cell_unit((e >> 14) & 7u, bias) * g.hf[1],
                                     cell_unit((e >> 17) & 7u, bias) * g.hf[2], dx, dy, dz);
            weights(gi, pi.w, lam, k, dx, dy, dz, d2, q < mine);
            tables();
            if (((q >> g.tsh) & 3) == 3) settle();
            e = nxt;
          }
          settle();
          if (SM::TURNS || s0 + ns >= n) store_tables();
        }
        for (int s0 = 0; s0 < n && !list_ok; s0 += ns) {
          // from the cells: a lane reads eight tables of each of its own pairs
          const int s = s0 + (tid >> g.tsh);
          for (int b = 0; b < nb; ++b) {
            float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (s < n) {
              const float4 gi = sm.gfe[s];
              const float fpi = sm.pos[s].w, lam = sm.rho[s];
              for_pairs(A, g, sm, s, t, T, [&](int k, float dx, float dy, float dz, float d2, uint32_t) {
                weights(gi, fpi, lam, k, dx, dy, dz, d2, true);
                const float4* const c = A.dtab + (size_t)rec.m[lane] * A.ktab + 8 * b;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                  const float4 f = q + 8 * b < A.nz2 ? rec.z[lane] : rec.r[lane];
                  a[q] = fmaf(c[q].x, f.x, fmaf(c[q].y, f.y, fmaf(c[q].z, f.z, fmaf(c[q].w, f.w, a[q]))));
                }
              });
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              double v = widen(a[q]);
#pragma unroll
              for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
#pragma unroll
              for (int bb = 0; bb < MAX_TABLES / 8; ++bb)
                if (bb == b && lane == q) accd[bb] += v;
            }
          }
          if (SM::TURNS || s0 + ns >= n) store_tables();
        }
        block_sums<MAX_TABLES>(sm, rows);
        if (tid < BMAX_PARAMS) {
          double v = row[11 + tid];
          for (int p = 0; p < A.nz2; ++p)
            if (A.pz2[p] == tid) v += sm.red[0][p];
          for (int p = 0; p < A.nrh; ++p)
            if (A.prh[p] == tid) v += sm.red[0][A.nz2 + p];
          row[11 + tid] = v;
        }
      }
    }
    block_sync();  // the next replica overwrites the shared memory
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
struct gbmd_batch {
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  std::string err;
  int nrep = 0;
  int64_t n = 0;
  int64_t *off = nullptr;
  double *lo = nullptr, *hi = nullptr, *L = nullptr, *x = nullptr, *y = nullptr, *z = nullptr;
  double *fx = nullptr, *fy = nullptr, *fz = nullptr, *ep = nullptr, *rep = nullptr;
  double *Ftx = nullptr, *Fty = nullptr, *Ftz = nullptr, *Et = nullptr;
  int *order = nullptr, *queue = nullptr, *d_err = nullptr;
  float4* tab = nullptr;
  float4* dtab = nullptr;
  BatchArgs a{};
  bool have_pot = false, have_targets = false;
  int block = 512, S = 1;
  int small_block = 0;           // threads per block of the small-replica kernel (0: by the number of replicas)
  cudaStream_t side = nullptr;   // runs the small-replica kernel beside the large one
  cudaEvent_t fork = nullptr, join = nullptr;
  int nbig = 0;                  // replicas of more than SMALL_ATOMS atoms (first in `order`)
  std::vector<int> rep_atoms;    // atoms per replica (host copy)
  uint32_t* nbl = nullptr;       // pair-list scratch of the large-replica kernel's blocks
  size_t nbl_regions = 0;
  uint32_t* nbl_small = nullptr; // and of the small-replica kernel's blocks
  size_t nbl_small_regions = 0;
  double* h_rows = nullptr;      // page-locked: the replicas' rows, then the error words
  cudaGraphExec_t graph = nullptr;
  int graph_adjoint = -1;
};

namespace {

int berr(gbmd_batch* b, int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  if (b) b->err = buf;
  return code;
}

#define BCUDA(b, call)                                                               \
  do {                                                                               \
    cudaError_t e_ = (call);                                                         \
    if (e_ != cudaSuccess) return berr((b), GBMD_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
  } while (0)

void free_atoms(gbmd_batch* b) {
  void* ps[] = {b->off, b->lo, b->hi, b->L, b->x, b->y, b->z, b->fx, b->fy, b->fz, b->ep, b->rep,
                b->Ftx, b->Fty, b->Ftz, b->Et, b->order};
  for (void* p : ps) cudaFree(p);
  if (b->h_rows) cudaFreeHost(b->h_rows);
  b->h_rows = nullptr;
  b->off = nullptr; b->lo = b->hi = b->L = b->x = b->y = b->z = nullptr;
  b->fx = b->fy = b->fz = b->ep = b->rep = nullptr;
  b->Ftx = b->Fty = b->Ftz = b->Et = nullptr;
  b->order = nullptr;
}

void drop_graph(gbmd_batch* b) {
  if (b->graph) cudaGraphExecDestroy(b->graph);
  b->graph = nullptr;
}

// spline a table of knot values and return its FP32 value coefficients
void table_f4(int n, double delta, const double* vals, double scale, std::vector<float4>& out) {
  std::vector<double> f(n + 1, 0.0), s((size_t)(n + 1) * 8);
  for (int k = 0; k < n; ++k) f[k + 1] = vals[k];
  gbmd::spline7(n, delta, f.data(), s.data());
  for (int m = 0; m <= n; ++m)
    out.push_back(make_float4((float)(s[m * 8 + 3] * scale), (float)(s[m * 8 + 4] * scale),
                              (float)(s[m * 8 + 5] * scale), (float)(s[m * 8 + 6] * scale)));
}

// 512 threads at most: large replicas at 128 registers (1,024 threads at 64:
// 4,480 against 4,340 us for 4,096 replicas of 32-2,048 atoms), small ones two
// blocks of 512 (or four of 256) per SM at 64 registers (one at 128: 210
// against 192 us for 256 replicas of 243 atoms).
constexpr int BIG_THREADS = 512, SMALL_THREADS = 512;
constexpr size_t SMEM_BIG = sizeof(SmemT<BMAX_ATOMS, BMAX_CELLS, BIG_THREADS>);
constexpr size_t SMEM_SMALL = sizeof(SmemT<SMALL_ATOMS, SMALL_CELLS, SMALL_THREADS>);
using BatchKernel = void (*)(BatchArgs);
BatchKernel big_kernel(int adjoint) {
  return adjoint ? &k_batch<BMAX_ATOMS, BMAX_CELLS, BIG_THREADS, 1, true>
                 : &k_batch<BMAX_ATOMS, BMAX_CELLS, BIG_THREADS, 1, false>;
}
BatchKernel small_kernel(int adjoint) {
  return adjoint ? &k_batch<SMALL_ATOMS, SMALL_CELLS, SMALL_THREADS, 2, true>
                 : &k_batch<SMALL_ATOMS, SMALL_CELLS, SMALL_THREADS, 2, false>;
}

// Threads per block of the small-replica kernel: with few replicas per SM,
// many threads (and lanes per atom) for each (256 replicas of 243 atoms, 512 /
// 256 / 128 threads: 192 / 211 / 307 us); with many, more blocks (4,000 of
// 32-500 atoms, 256 / 128: 1,558 / 1,832 us).
int small_threads(const gbmd_batch* b) {
  if (b->small_block) return b->small_block;
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->device);
  return b->nrep - b->nbig <= 4 * sms ? 512 : 256;
}

}  // namespace

extern "C" {

int gbmd_batch_create(gbmd_batch** out, int device, void* stream) {
  if (!out) return GBMD_ERR_INVALID;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return GBMD_ERR_NO_DEVICE;
  if (device < 0 || device >= ndev) return GBMD_ERR_INVALID;
  gbmd_batch* b = new gbmd_batch();
  b->device = device;
  cudaSetDevice(device);
  if (stream) {
    b->stream = (cudaStream_t)stream;
  } else {
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess) {
      delete b;
      return GBMD_ERR_CUDA;
    }
    b->own_stream = true;
  }
  if (cudaMalloc(&b->queue, sizeof(int) * 2) != cudaSuccess || cudaMalloc(&b->d_err, sizeof(int) * 4) != cudaSuccess ||
      cudaMemset(b->d_err, 0, sizeof(int) * 4) != cudaSuccess ||
      cudaFuncSetAttribute(big_kernel(0), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BIG) != cudaSuccess ||
      cudaFuncSetAttribute(big_kernel(1), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BIG) != cudaSuccess ||
      cudaFuncSetAttribute(small_kernel(0), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_SMALL) != cudaSuccess ||
      cudaFuncSetAttribute(small_kernel(1), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_SMALL) != cudaSuccess ||
      cudaStreamCreateWithFlags(&b->side, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&b->join, cudaEventDisableTiming) != cudaSuccess) {
    cudaFree(b->queue);
    cudaFree(b->d_err);
    if (b->side) cudaStreamDestroy(b->side);
    if (b->fork) cudaEventDestroy(b->fork);
    if (b->join) cudaEventDestroy(b->join);
    if (b->own_stream) cudaStreamDestroy(b->stream);
    delete b;
    return GBMD_ERR_CUDA;
  }
  *out = b;
  return GBMD_OK;
}

int gbmd_batch_destroy(gbmd_batch* b) {
  if (!b) return GBMD_OK;
  cudaSetDevice(b->device);
  if (b->stream) cudaStreamSynchronize(b->stream);
  drop_graph(b);
  free_atoms(b);
  cudaFree(b->queue);
  cudaFree(b->d_err);
  cudaFree(b->tab);
  cudaFree(b->dtab);
  cudaFree(b->nbl);
  cudaFree(b->nbl_small);
  if (b->side) cudaStreamDestroy(b->side);
  if (b->fork) cudaEventDestroy(b->fork);
  if (b->join) cudaEventDestroy(b->join);
  if (b->own_stream) cudaStreamDestroy(b->stream);
  delete b;
  return GBMD_OK;
}

const char* gbmd_batch_last_error(const gbmd_batch* b) { return b ? b->err.c_str() : "null batch"; }

int gbmd_batch_set_eam_alloy(gbmd_batch* b, int nrho, double drho, int nr, double dr, const double* frho,
                             const double* rhor, const double* z2r, double rcut, double conv_z2r,
                             double conv_frho) {
  if (!b || nrho < 5 || nr < 5 || !(drho > 0) || !(dr > 0) || !frho || !rhor || !z2r || !(rcut > 0))
    return berr(b, GBMD_ERR_INVALID, "bad eam_alloy tables");
  std::vector<float4> h, z;
  // rho' coefficients (3c3, 2c4, c5) / dr beside the pair function's, so that
  // the force pass reads one 32-byte knot
  table_f4(nr, dr, z2r, conv_z2r, z);
  {
    std::vector<double> f(nr + 1, 0.0), s((size_t)(nr + 1) * 8);
    for (int k = 0; k < nr; ++k) f[k + 1] = rhor[k];
    gbmd::spline7(nr, dr, f.data(), s.data());
    for (int m = 0; m <= nr; ++m) {
      h.push_back(make_float4((float)(3.0 * s[m * 8 + 3] / dr), (float)(2.0 * s[m * 8 + 4] / dr),
                              (float)(s[m * 8 + 5] / dr), 0.f));
      h.push_back(z[m]);
    }
  }
  table_f4(nrho, drho, frho, conv_frho, h);
  table_f4(nr, dr, rhor, 1.0, h);
  cudaSetDevice(b->device);
  cudaFree(b->tab);
  b->tab = nullptr;
  BCUDA(b, cudaMalloc(&b->tab, sizeof(float4) * h.size()));
  BCUDA(b, cudaMemcpy(b->tab, h.data(), sizeof(float4) * h.size(), cudaMemcpyHostToDevice));
  BatchArgs& A = b->a;
  A.fz8 = b->tab;
  A.frho4 = A.fz8 + 2 * (nr + 1);
  A.rhor4 = A.frho4 + (nrho + 1);
  A.nr = nr;
  A.nrho = nrho;
  A.rdr = (float)(1.0 / dr);
  A.rdrho = (float)(1.0 / drho);
  A.rhomax = (float)((nrho - 1) * drho);
  A.rcut = rcut;
  A.rcut2 = rcut * rcut;
  b->have_pot = true;
  A.nz2 = A.nrh = A.nfr = A.ktab = 0;
  drop_graph(b);
  return GBMD_OK;
}

int gbmd_batch_set_param_derivatives(gbmd_batch* b, int nparam, const double* dfrho, const double* drhor,
                                     const double* dz2r, double conv_z2r, double conv_frho) {
  if (!b || !b->have_pot || nparam < 1 || nparam > BMAX_PARAMS || !dfrho || !drhor || !dz2r)
    return berr(b, GBMD_ERR_INVALID, "bad parameter derivative tables (set the potential first)");
  BatchArgs& A = b->a;
  const int nr = A.nr, nrho = A.nrho;
  const double dr = 1.0 / (double)A.rdr, drho = 1.0 / (double)A.rdrho;
  std::vector<float4> fr, rh, zz;
  A.nz2 = A.nrh = A.nfr = 0;
  for (int p = 0; p < nparam; ++p) {
    auto nonzero = [](const double* v, int k) {
      for (int q = 0; q < k; ++q)
        if (v[q] != 0.0) return true;
      return false;
    };
    if (nonzero(dfrho + (size_t)p * nrho, nrho)) {
      table_f4(nrho, drho, dfrho + (size_t)p * nrho, conv_frho, fr);
      A.pfr[A.nfr++] = p;
    }
    if (nonzero(drhor + (size_t)p * nr, nr)) {
      table_f4(nr, dr, drhor + (size_t)p * nr, 1.0, rh);
      A.prh[A.nrh++] = p;
    }
    if (nonzero(dz2r + (size_t)p * nr, nr)) {
      table_f4(nr, dr, dz2r + (size_t)p * nr, conv_z2r, zz);
      A.pz2[A.nz2++] = p;
    }
  }
  // the pair tables knot by knot, a multiple of eight of them
  A.ktab = (A.nz2 + A.nrh + 7) / 8 * 8;
  std::vector<float4> h;
  for (int m = 0; m <= nr; ++m)
    for (int k = 0; k < A.ktab; ++k) {
      if (k < A.nz2) h.push_back(zz[(size_t)k * (nr + 1) + m]);
      else if (k < A.nz2 + A.nrh) h.push_back(rh[(size_t)(k - A.nz2) * (nr + 1) + m]);
      else h.push_back(make_float4(0.f, 0.f, 0.f, 0.f));
    }
  const size_t pair_tables = h.size();
  h.insert(h.end(), fr.begin(), fr.end());
  cudaSetDevice(b->device);
  cudaFree(b->dtab);
  b->dtab = nullptr;
  BCUDA(b, cudaMalloc(&b->dtab, sizeof(float4) * (h.size() + 1)));
  BCUDA(b, cudaMemcpy(b->dtab, h.data(), sizeof(float4) * h.size(), cudaMemcpyHostToDevice));
  A.dtab = b->dtab;
  A.dfrho4 = A.dtab + pair_tables;
  drop_graph(b);
  return GBMD_OK;
}

int gbmd_batch_upload(gbmd_batch* b, int nrep, const int64_t* offsets, const double* lo, const double* hi,
                      const double* x, const double* y, const double* z) {
  if (!b || nrep < 1 || !offsets || !lo || !hi || !x || !y || !z) return berr(b, GBMD_ERR_INVALID, "bad replicas");
  if (offsets[0] != 0) return berr(b, GBMD_ERR_INVALID, "offsets[0] must be 0");
  for (int r = 0; r < nrep; ++r) {
    const int64_t m = offsets[r + 1] - offsets[r];
    if (m < 0) return berr(b, GBMD_ERR_INVALID, "offsets must be non-decreasing");
    if (m > BMAX_ATOMS) return berr(b, GBMD_ERR_TOO_LARGE, "replica %d has %lld atoms (max %d)", r, (long long)m, BMAX_ATOMS);
    if (!gbmd::batch_box_ok(lo + 3 * r, hi + 3 * r))
      return berr(b, GBMD_ERR_INVALID, "replica %d: empty or non-finite box", r);
  }
  cudaSetDevice(b->device);
  cudaStreamSynchronize(b->stream);
  drop_graph(b);
  free_atoms(b);
  const int64_t n = offsets[nrep];
  b->nrep = nrep;
  b->n = n;
  std::vector<double> L(3 * (size_t)nrep);
  for (size_t q = 0; q < L.size(); ++q) L[q] = hi[q] - lo[q];
  // largest replicas first (longest-processing-time order for the queue)
  std::vector<int> ord(nrep);
  std::iota(ord.begin(), ord.end(), 0);
  std::stable_sort(ord.begin(), ord.end(), [&](int a, int c) {
    return offsets[a + 1] - offsets[a] > offsets[c + 1] - offsets[c];
  });
  b->rep_atoms.resize(nrep);
  b->nbig = 0;
  for (int r = 0; r < nrep; ++r) {
    b->rep_atoms[r] = (int)(offsets[r + 1] - offsets[r]);
    if (b->rep_atoms[r] > SMALL_ATOMS) ++b->nbig;
  }
  const size_t nb = sizeof(double) * (size_t)(n > 0 ? n : 1);
  BCUDA(b, cudaMalloc(&b->off, sizeof(int64_t) * (nrep + 1)));
  BCUDA(b, cudaMalloc(&b->lo, sizeof(double) * 3 * nrep));
  BCUDA(b, cudaMalloc(&b->L, sizeof(double) * 3 * nrep));
  BCUDA(b, cudaMalloc(&b->hi, sizeof(double) * 3 * nrep));
  BCUDA(b, cudaMalloc(&b->order, sizeof(int) * nrep));
  BCUDA(b, cudaMalloc(&b->rep, sizeof(double) * REP_ROW * nrep));
  BCUDA(b, cudaMallocHost(&b->h_rows, sizeof(double) * ((size_t)REP_ROW * nrep + 2)));
  double** arrs[] = {&b->x, &b->y, &b->z, &b->fx, &b->fy, &b->fz, &b->ep, &b->Ftx, &b->Fty, &b->Ftz, &b->Et};
  for (double** p : arrs) BCUDA(b, cudaMalloc(p, nb));
  BCUDA(b, cudaMemcpy(b->off, offsets, sizeof(int64_t) * (nrep + 1), cudaMemcpyHostToDevice));
  BCUDA(b, cudaMemcpy(b->lo, lo, sizeof(double) * 3 * nrep, cudaMemcpyHostToDevice));
  BCUDA(b, cudaMemcpy(b->L, L.data(), sizeof(double) * 3 * nrep, cudaMemcpyHostToDevice));
  BCUDA(b, cudaMemcpy(b->hi, hi, sizeof(double) * 3 * nrep, cudaMemcpyHostToDevice));
  BCUDA(b, cudaMemcpy(b->order, ord.data(), sizeof(int) * nrep, cudaMemcpyHostToDevice));
  BCUDA(b, cudaMemcpy(b->x, x, nb, cudaMemcpyHostToDevice));
  BCUDA(b, cudaMemcpy(b->y, y, nb, cudaMemcpyHostToDevice));
  BCUDA(b, cudaMemcpy(b->z, z, nb, cudaMemcpyHostToDevice));
  b->have_targets = false;
  return GBMD_OK;
}

int gbmd_batch_set_targets(gbmd_batch* b, const double* fx, const double* fy, const double* fz, const double* e,
                           double wF, double wE) {
  if (!b || !b->x || !fx || !fy || !fz || !e) return berr(b, GBMD_ERR_INVALID, "bad targets (upload first)");
  const size_t nb = sizeof(double) * (size_t)b->n;
  BCUDA(b, cudaMemcpy(b->Ftx, fx, nb, cudaMemcpyHostToDevice));
  BCUDA(b, cudaMemcpy(b->Fty, fy, nb, cudaMemcpyHostToDevice));
  BCUDA(b, cudaMemcpy(b->Ftz, fz, nb, cudaMemcpyHostToDevice));
  BCUDA(b, cudaMemcpy(b->Et, e, nb, cudaMemcpyHostToDevice));
  b->a.wF = wF;
  b->a.wE = wE;
  b->have_targets = true;
  drop_graph(b);
  return GBMD_OK;
}

int gbmd_batch_set_small_block(gbmd_batch* b, int block) {
  if (!b || block < 64 || block > 256 || block % 32) return berr(b, GBMD_ERR_INVALID, "small block in [64,256], multiple of 32");
  b->small_block = block;
  drop_graph(b);
  return GBMD_OK;
}

int gbmd_batch_set_small_block_auto(gbmd_batch* b) {
  if (!b) return GBMD_ERR_INVALID;
  b->small_block = 0;
  drop_graph(b);
  return GBMD_OK;
}

int gbmd_batch_set_launch(gbmd_batch* b, int block, int stencil) {
  if (!b || block < 64 || block > 512 || block % 32 || (stencil != 1 && stencil != 2))
    return berr(b, GBMD_ERR_INVALID, "block in [64,512] (multiple of 32), stencil 1 or 2");
  b->block = block;
  b->S = stencil;
  drop_graph(b);
  return GBMD_OK;
}

// Blocks of a persistent launch: as many as fit on the device at once, at
// most one per replica of its queue.  big: the large-replica kernel (the
// autotuned block), else the small-replica kernel (b->small_block threads).
static int persistent_grid(gbmd_batch* b, bool big, int adjoint) {
  int dev_sms = 0, per_sm = 0;
  cudaDeviceGetAttribute(&dev_sms, cudaDevAttrMultiProcessorCount, b->device);
  if (big)
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, big_kernel(adjoint), b->block, SMEM_BIG);
  else
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, small_kernel(adjoint), small_threads(b), SMEM_SMALL);
  const int nq = big ? b->nbig : b->nrep - b->nbig;
  return std::max(1, std::min(nq, dev_sms * std::max(per_sm, 1)));
}

// pair-list scratch for `regions` blocks of each kernel (allocated outside any capture)
static int ensure_nbl(gbmd_batch* b, int regions, int small_regions) {
  if ((size_t)regions > b->nbl_regions) {
    drop_graph(b);
    cudaFree(b->nbl);
    b->nbl = nullptr;
    b->nbl_regions = 0;
    BCUDA(b, cudaMalloc(&b->nbl, sizeof(uint32_t) * BMAX_ATOMS * NBL_MAX * (size_t)regions));
    b->nbl_regions = (size_t)regions;
  }
  if ((size_t)small_regions > b->nbl_small_regions) {
    drop_graph(b);
    cudaFree(b->nbl_small);
    b->nbl_small = nullptr;
    b->nbl_small_regions = 0;
    BCUDA(b, cudaMalloc(&b->nbl_small, sizeof(uint32_t) * SMALL_ATOMS * NBL_MAX * (size_t)small_regions));
    b->nbl_small_regions = (size_t)small_regions;
  }
  return GBMD_OK;
}

// Replicas of more than SMALL_ATOMS atoms run in the large-replica kernel
// (blocks of up to 512 threads), the rest in the small-replica kernel (64-512
// threads, less shared memory, several blocks per SM); each takes its
// replicas from its own queue, largest first.
static int batch_launch(gbmd_batch* b, int adjoint, int per_replica) {
  BatchArgs A = b->a;
  A.nrep = b->nrep;
  A.off = b->off;
  A.lo = b->lo;
  A.hi = b->hi;
  A.L = b->L;
  A.x = b->x; A.y = b->y; A.z = b->z;
  A.fx = b->fx; A.fy = b->fy; A.fz = b->fz; A.ep = b->ep;
  A.rep = b->rep;
  A.order = b->order;
  A.queue = b->queue;
  A.err = b->d_err;
  A.S = b->S;
  A.Ftx = b->Ftx; A.Fty = b->Fty; A.Ftz = b->Ftz; A.Et = b->Et;
  if (per_replica) {
    for (int r = 0; r < b->nrep; ++r) {
      A.single = r;
      if (b->rep_atoms[r] > SMALL_ATOMS) {
        A.nbl = b->nbl;
        big_kernel(adjoint)<<<1, b->block, SMEM_BIG, b->stream>>>(A);
      } else {
        A.nbl = b->nbl_small;
        small_kernel(adjoint)<<<1, small_threads(b), SMEM_SMALL, b->stream>>>(A);
      }
    }
  } else {
    A.single = -1;
    BCUDA(b, cudaMemsetAsync(b->queue, 0, sizeof(int) * 2, b->stream));
    // the two size classes on two streams, so the small-replica blocks take
    // over SMs as the large-replica kernel's blocks run out of work
    const bool both = b->nbig > 0 && b->nrep > b->nbig;
    if (both) {
      BCUDA(b, cudaEventRecord(b->fork, b->stream));
      BCUDA(b, cudaStreamWaitEvent(b->side, b->fork, 0));
    }
    if (b->nbig > 0) {
      const int grid = persistent_grid(b, true, adjoint);
      if ((size_t)grid > b->nbl_regions) return berr(b, GBMD_ERR_INVALID, "pair-list scratch not sized");
      BatchArgs Ab = A;
      Ab.nrep = b->nbig;
      Ab.nbl = b->nbl;
      big_kernel(adjoint)<<<grid, b->block, SMEM_BIG, b->stream>>>(Ab);
    }
    if (b->nrep > b->nbig) {
      const int grid = persistent_grid(b, false, adjoint);
      if ((size_t)grid > b->nbl_small_regions) return berr(b, GBMD_ERR_INVALID, "pair-list scratch not sized");
      BatchArgs As = A;
      As.nrep = b->nrep - b->nbig;
      As.order = b->order + b->nbig;
      As.queue = b->queue + 1;
      As.nbl = b->nbl_small;
      small_kernel(adjoint)<<<grid, small_threads(b), SMEM_SMALL, both ? b->side : b->stream>>>(As);
    }
    if (both) {
      BCUDA(b, cudaEventRecord(b->join, b->side));
      BCUDA(b, cudaStreamWaitEvent(b->stream, b->join, 0));
    }
  }
  BCUDA(b, cudaGetLastError());
  return GBMD_OK;
}

int gbmd_batch_run(gbmd_batch* b, int adjoint, int per_replica, int use_graph) {
  if (!b || !b->have_pot || !b->x) return berr(b, GBMD_ERR_INVALID, "set the potential and upload replicas first");
  if (adjoint && (!b->have_targets || b->a.nz2 + b->a.nrh + b->a.nfr == 0))
    return berr(b, GBMD_ERR_INVALID, "adjoint needs targets and parameter derivatives");
  cudaSetDevice(b->device);
  {
    const int rc = per_replica ? ensure_nbl(b, 1, 1)
                               : ensure_nbl(b, b->nbig > 0 ? persistent_grid(b, true, adjoint) : 0,
                                            b->nrep > b->nbig ? persistent_grid(b, false, adjoint) : 0);
    if (rc) return rc;
  }
  if (use_graph && !per_replica) {
    if (!b->graph || b->graph_adjoint != adjoint) {
      drop_graph(b);
      cudaGraph_t g;
      BCUDA(b, cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
      const int rc = batch_launch(b, adjoint, 0);
      cudaError_t e = cudaStreamEndCapture(b->stream, &g);
      if (rc) return rc;
      if (e != cudaSuccess) return berr(b, GBMD_ERR_CUDA, "capture: %s", cudaGetErrorString(e));
      e = cudaGraphInstantiate(&b->graph, g, 0);
      cudaGraphDestroy(g);
      if (e != cudaSuccess) return berr(b, GBMD_ERR_CUDA, "instantiate: %s", cudaGetErrorString(e));
      b->graph_adjoint = adjoint;
    }
    BCUDA(b, cudaGraphLaunch(b->graph, b->stream));
  } else {
    const int rc = batch_launch(b, adjoint, per_replica);
    if (rc) return rc;
  }
  return GBMD_OK;
}

int gbmd_batch_synchronize(gbmd_batch* b) {
  if (!b) return GBMD_ERR_INVALID;
  BCUDA(b, cudaStreamSynchronize(b->stream));
  int h[4];
  BCUDA(b, cudaMemcpy(h, b->d_err, sizeof(h), cudaMemcpyDeviceToHost));
  if (h[0] & 16) return berr(b, GBMD_ERR_TOO_LARGE, "a replica exceeded the per-block limits (atoms or box)");
  return GBMD_OK;
}

int gbmd_batch_download(gbmd_batch* b, double* fx, double* fy, double* fz, double* ep, double* rep_energy,
                        double* rep_virial, double* loss, double* grad) {
  if (!b || !b->x) return GBMD_ERR_INVALID;
  // everything queued behind the run, one wait at the end
  cudaSetDevice(b->device);
  const size_t nb = sizeof(double) * (size_t)b->n, nrow = (size_t)REP_ROW * b->nrep;
  double* const rows = b->h_rows;
  int* const err = reinterpret_cast<int*>(rows + nrow);
  BCUDA(b, cudaMemcpyAsync(rows, b->rep, sizeof(double) * nrow, cudaMemcpyDeviceToHost, b->stream));
  BCUDA(b, cudaMemcpyAsync(err, b->d_err, sizeof(int) * 4, cudaMemcpyDeviceToHost, b->stream));
  if (fx) BCUDA(b, cudaMemcpyAsync(fx, b->fx, nb, cudaMemcpyDeviceToHost, b->stream));
  if (fy) BCUDA(b, cudaMemcpyAsync(fy, b->fy, nb, cudaMemcpyDeviceToHost, b->stream));
  if (fz) BCUDA(b, cudaMemcpyAsync(fz, b->fz, nb, cudaMemcpyDeviceToHost, b->stream));
  if (ep) BCUDA(b, cudaMemcpyAsync(ep, b->ep, nb, cudaMemcpyDeviceToHost, b->stream));
  BCUDA(b, cudaStreamSynchronize(b->stream));
  if (err[0] & 16) return berr(b, GBMD_ERR_TOO_LARGE, "a replica exceeded the per-block limits (atoms or box)");
  double L = 0.0, G[BMAX_PARAMS] = {0};
  for (int r = 0; r < b->nrep; ++r) {  // replica order: fixed summation order
    const double* row = &rows[(size_t)r * REP_ROW];
    if (rep_energy) rep_energy[r] = row[0];
    if (rep_virial)
      for (int q = 0; q < 9; ++q) rep_virial[9 * r + q] = row[1 + q];
    L += row[10];
    for (int q = 0; q < BMAX_PARAMS; ++q) G[q] += row[11 + q];
  }
  if (loss) *loss = L;
  if (grad)
    for (int q = 0; q < BMAX_PARAMS; ++q) grad[q] = G[q];
  return GBMD_OK;
}

}  // extern "C"
