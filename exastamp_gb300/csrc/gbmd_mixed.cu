// gbmd_mixed.cu -- mixed-precision pair kernels (FP32 pair arithmetic, FP64
// state) for sm_103a: lj_compute_force / lj_multi_force, and the eam_alloy
// density+embedding and force passes.
//
// Same functions as the FP64 kernels (lennard_jones.h L41-50,
// force_op_impl2.hxx L33-68, pair_potential_force_op_multiparam.h L92-118,
// eam_alloy.h L198-313, eam_force_op_multimat.h L114-343), evaluated on
// home-cell-relative FP32 coordinates: dr = (p_j - p_i) + s*h with s the
// stencil offset of j's cell, exact to ~1e-7 relative.  Forces, densities
// and energies are summed with compensated (Kahan) FP32 sums; per-atom
// results are converted to FP64 once.  Cutoff membership matches FP64
// exactly: pairs with FP32 d2 within band_tol of rcut are re-tested in FP64.
//
// Loop structure: each lane reads V list entries with one coalesced load
// (V = 4: 16 B per lane, streamed past L1 so the gathers keep it), the next
// row already in flight; per entry one 16 B position gather (single-element
// EAM force pass: the position carries F'(rho_j) in w), one 16 B spline-knot
// gather per table; branch-free except the rare FP64 re-test.  The V terms
// of a row are added in FP32, the row sum goes into the compensated sum.
// 1/r and r come from one rsqrt; the stencil offset decodes to an exact
// float in two integer/FP ops per axis.
#include <algorithm>
#include <cmath>

#include "gbmd_pair_common.cuh"

namespace gbmd {

// Two list entries at once in packed FP32 (sm_100 float2 arithmetic: one
// instruction per pair of lanes' worth of FADD / FMUL / FFMA).  Each half is
// geom_f of its entry, operation for operation: (p_j - p_i) is p_j + (-p_i),
// which rounds identically.  npi = (-p_i) in both halves of each axis.
struct GeomF2 {
  float2 dx, dy, dz, d2;
};

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

__device__ __forceinline__ GeomF2 geom_f2(uint32_t ea, uint32_t eb, const float4& pa, const float4& pb,
                                          const float2& npx, const float2& npy, const float2& npz, const float2& hx,
                                          const float2& hy, const float2& hz) {
  GeomF2 r;
  r.dx = __ffma2_rn(f2(twice_dx(ea), twice_dx(eb)), hx, __fadd2_rn(f2(pa.x, pb.x), npx));
  r.dy = __ffma2_rn(f2(twice_dy(ea), twice_dy(eb)), hy, __fadd2_rn(f2(pa.y, pb.y), npy));
  r.dz = __ffma2_rn(f2(twice_dz(ea), twice_dz(eb)), hz, __fadd2_rn(f2(pa.z, pb.z), npz));
  r.d2 = __ffma2_rn(r.dx, r.dx, __ffma2_rn(r.dy, r.dy, __fmul2_rn(r.dz, r.dz)));
  return r;
}

// The per-atom constants of geom_f2: -p_i and the cell edges, packed.
struct PairFrame {
  float2 npx, npy, npz, hx, hy, hz;
  __device__ __forceinline__ PairFrame(const float4& pi, const Grid& g)
      : npx(f2(-pi.x, -pi.x)), npy(f2(-pi.y, -pi.y)), npz(f2(-pi.z, -pi.z)), hx(f2(g.hh[0], g.hh[0])),
        hy(f2(g.hh[1], g.hh[1])), hz(f2(g.hh[2], g.hh[2])) {}
  __device__ __forceinline__ GeomF2 geom(uint32_t ea, uint32_t eb, const float4& pa, const float4& pb) const {
    return geom_f2(ea, eb, pa, pb, npx, npy, npz, hx, hy, hz);
  }
};

__device__ __forceinline__ void reduce6(float* v, int T) {
  for (int off = T / 2; off > 0; off >>= 1)
#pragma unroll
    for (int q = 0; q < 6; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], off);
}

__device__ __forceinline__ void vir9(const float* v, double* o) {
  // symmetric pair virial: xx yy zz xy xz yz -> row-major 3x3
  o[0] = v[0]; o[1] = v[3]; o[2] = v[4];
  o[3] = v[3]; o[4] = v[1]; o[5] = v[5];
  o[6] = v[4]; o[7] = v[5]; o[8] = v[2];
}

// Atom i's list as the T lanes of its group read it: entry k = r*T*V + q*T +
// lane is lane `lane`'s q-th of row r (see list_word), so that one gather of
// the group touches T consecutive entries, which lie in the same one or two
// cells and mostly in the same 128-byte lines.  A warp's position gather
// touches 16.5 lines with one lane per atom, 12.0 with two and 8.7 with four
// (Cu crystal, counted), and the L1 takes about a cycle for each.  A row's V
// entries are one load that bypasses L1 (each entry is used once per kernel).
// Entries at or beyond nn, in the last row only, are replaced by a harmless
// stand-in: j = i seen through the +x stencil offset, a separation of one
// cell edge (>= rcut + skin), which no cutoff test accepts.
template <int T, int V>
struct ListRows {
  static constexpr int W = T * V;
  const uint32_t* p;  // nbr + i*W + lane*V
  int64_t stride;
  int nrow, nfull, rem, lane, nn;
  uint32_t standin;
  __device__ __forceinline__ ListRows(const uint32_t* nbr, int64_t i, int lane_, int64_t stride_, int nn_)
      : p(nbr + (size_t)i * W + lane_ * V), stride(stride_), lane(lane_), nn(nn_) {
    nrow = (nn + W - 1) / W;
    nfull = nn / W;
    rem = nn - nfull * W;
    standin = (uint32_t)i | (code_of(1, 0, 0) << GBMD_IDX_BITS);
  }
  __device__ __forceinline__ void load(int r, uint32_t (&e)[V]) const {
    const uint32_t* q = p + (size_t)r * stride;
    if constexpr (V == 4) {
      // read once per kernel: keep it out of L1, which serves the gathers
      asm("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
          : "=r"(e[0]), "=r"(e[1]), "=r"(e[2]), "=r"(e[3])
          : "l"(q));
    } else {
#pragma unroll
      for (int v = 0; v < V; ++v) e[v] = __ldcs(q + v);
    }
  }
  __device__ __forceinline__ bool valid(int r, int q) const { return r * W + q * T + lane < nn; }
  __device__ __forceinline__ bool in_tail(int q) const { return q * T + lane < rem; }
};

// body(entries, valid): every row of L in order, N = V entries of a full row
// or N = V / 2 (at least one) of the last, partial one, which stops after
// the half that holds its last entry.
template <int N>
struct RowPart {
  uint32_t e[N];
  bool ok[N];
  size_t at;  // the first entry's word, from the lane's first
};

template <int T, int V, class Body>
__device__ __forceinline__ void for_rows(const ListRows<T, V>& L, Body body) {
  constexpr int H = V >= 2 ? V / 2 : 1;
  uint32_t ent[V], nxt[V];
  if (L.nrow > 0) L.load(0, ent);
  for (int r = 0; r < L.nfull; ++r) {
    if (r + 1 < L.nrow) L.load(r + 1, nxt);
    RowPart<V> P;
    P.at = (size_t)r * L.stride;
#pragma unroll
    for (int q = 0; q < V; ++q) {
      P.e[q] = ent[q];
      P.ok[q] = true;
    }
    body(P);
#pragma unroll
    for (int q = 0; q < V; ++q) ent[q] = nxt[q];
  }
#pragma unroll
  for (int h = 0; h < V; h += H) {
    if (L.rem > h * T) {
      RowPart<H> P;
      P.at = (size_t)L.nfull * L.stride + h;
#pragma unroll
      for (int q = 0; q < H; ++q) {
        P.ok[q] = L.in_tail(h + q);
        P.e[q] = P.ok[q] ? ent[h + q] : L.standin;
      }
      body(P);
    }
  }
}

// ---------------------------------------------------------------------------
// Neighbour-position sources.  GlobalFetch gathers position j from the
// cell-sorted array; StagedFetch reads it from the block's shared-memory copy
// of the cells around its home cells (see stage_cells): the list entry's
// stencil row (dy, dz) picks one of nine staged row segments, each at most
// two contiguous global ranges (a row wraps at most once in x).
// ---------------------------------------------------------------------------
struct GlobalFetch {
  const float4* __restrict__ P;
  __device__ __forceinline__ float4 operator()(uint32_t ent, uint32_t j) const {
    float4 v;
    asm("ld.global.nc.L1::evict_last.v4.f32 {%0,%1,%2,%3}, [%4];"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
        : "l"(P + j));
    return v;
  }
};

struct StagedFetch {
  const float4* pos;   // staged positions (shared memory)
  const int4* rows;    // 16 entries by the entry's bits of dy, dz: {delta0, g1, n1, delta1}
  __device__ __forceinline__ float4 operator()(uint32_t ent, uint32_t j) const {
    const int4 t = rows[(ent >> 28) & 15u];
    const int jj = (int)j;
    const int slot = jj - ((unsigned)(jj - t.y) < (unsigned)t.z ? t.w : t.x);
    return pos[slot];
  }
};

// Stage, for the block's K home cells (x0 .. x0+K-1 of row (y, z), taken
// from blockIdx), the positions of every atom of the cells x0-1 .. x0+K in
// the nine rows (y+dy, z+dz) into `pos` and the translation table into
// `rows`; a0 / a1 receive the block's home atom range.  Returns false (then
// the block gathers from global memory) when they exceed `cap` atoms.
__device__ bool stage_cells(const Grid& g, const int32_t* __restrict__ cstart, const float4* __restrict__ src,
                            int K, int cap, float4* pos, int4* rows, int* sh, int64_t& a0, int64_t& a1) {
  const int ncx = g.nc[0], ncy = g.nc[1], ncz = g.nc[2];
  const int x0 = blockIdx.x * K, y = blockIdx.y, z = blockIdx.z;
  const int x1 = min(x0 + K, ncx);  // exclusive
  const int64_t rowbase = ((int64_t)z * ncy + y) * ncx;
  a0 = cstart[rowbase + x0];
  a1 = cstart[rowbase + x1];
  // sh[0..35]: per row s = 0..8, global start / count of range A and B
  if (threadIdx.x < 9) {
    const int s = threadIdx.x, dy = s % 3 - 1, dz = s / 3 - 1;
    const int yy = (y + dy + ncy) % ncy, zz = (z + dz + ncz) % ncz;
    const int64_t rb = ((int64_t)zz * ncy + yy) * ncx;
    int la = 0, ha = ncx - 1, lb = 0, hb = -1;  // inclusive cell ranges; B empty
    if (ncx > x1 - x0 + 2) {
      const int xs = x0 - 1, xe = x1;
      if (xs < 0) { la = ncx - 1; ha = ncx - 1; lb = 0; hb = xe; }
      else if (xe >= ncx) { la = xs; ha = ncx - 1; lb = 0; hb = 0; }
      else { la = xs; ha = xe; }
    }
    const int ga = cstart[rb + la], na = cstart[rb + ha + 1] - ga;
    const int gb = hb >= lb ? cstart[rb + lb] : 0, nb = hb >= lb ? cstart[rb + hb + 1] - gb : 0;
    sh[4 * s] = ga; sh[4 * s + 1] = na; sh[4 * s + 2] = gb; sh[4 * s + 3] = nb;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int off = 0;
    for (int q = 0; q < 16; ++q) rows[q] = make_int4(0, 0, 0, 0);
    for (int s = 0; s < 9; ++s) {
      const int ga = sh[4 * s], na = sh[4 * s + 1], gb = sh[4 * s + 2], nb = sh[4 * s + 3];
      const int oa = off, ob = off + na;
      off += na + nb;
      const int key = (int)code_of(s % 3 - 1, s / 3 - 1, 0);
      rows[key] = make_int4(ga - oa, gb, nb, gb - ob);
      sh[36 + 2 * s] = oa;
      sh[36 + 2 * s + 1] = ob;
    }
    sh[54] = off;
  }
  __syncthreads();
  const int total = sh[54];
  if (total > cap) return false;  // uniform
  // all copies in flight at once: slot u belongs to the last segment starting
  // at or before it (18 segments A0 B0 A1 B1 ... in staging order)
  for (int u = threadIdx.x; u < total; u += blockDim.x) {
    int seg = 0;
#pragma unroll
    for (int q = 1; q < 18; ++q)
      if (sh[36 + q] <= u) seg = q;
    const int s = seg >> 1, b = seg & 1;
    const int g0 = sh[4 * s + 2 * b];
    const float4* from = &src[g0 + (u - sh[36 + seg])];
    const unsigned to = (unsigned)__cvta_generic_to_shared(&pos[u]);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(to), "l"(from) : "memory");
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  return true;
}

// ---------------------------------------------------------------------------
// Lennard-Jones
// ---------------------------------------------------------------------------
struct LJF {
  float sig2, eps24, eps4, ecut, rc2lo, rc2hi;
  double rc2, rc;
};

struct LJTabSmem {
  float4 a[GBMD_MAX_TYPES * GBMD_MAX_TYPES];   // sig2, eps24, eps4, ecut
  float2 b[GBMD_MAX_TYPES * GBMD_MAX_TYPES];   // rc2lo, rc2hi
  double r[GBMD_MAX_TYPES * GBMD_MAX_TYPES];   // rc
};

__device__ __forceinline__ void lj_load_table(LJTabSmem& t, const LJPair* __restrict__ tab, int ntypes) {
  for (int q = threadIdx.x; q < ntypes * ntypes; q += blockDim.x) {
    const LJPair& p = tab[q];
    t.a[q] = make_float4(p.sig2f, p.eps24f, p.eps4f, p.ecutf);
    t.b[q] = make_float2(p.rc2lo, p.rc2hi);
    t.r[q] = p.rc;
  }
  __syncthreads();
}

// geom_f with the stencil offset through the 2^23 mantissa trick, an FP32
// addition an axis in place of geom_f's second integer instruction: for the
// kernels that the L1 data path or registers bound, not instruction issue
// (LJ mixtures without energies; one-element bond passes: 4M atoms 1,197
// against 1,224 us with geom_f).
__device__ __forceinline__ float unit_of(uint32_t b) { return __int_as_float((b & 3u) ^ 0x4b000002u) - 8388610.0f; }

__device__ __forceinline__ GeomF geom_u(uint32_t ent, const float4& pj, const float4& pi, const Grid& g) {
  GeomF r;
  r.dx = fmaf(unit_of(ent >> 26), g.hf[0], pj.x - pi.x);
  r.dy = fmaf(unit_of(ent >> 28), g.hf[1], pj.y - pi.y);
  r.dz = fmaf(unit_of(ent >> 30), g.hf[2], pj.z - pi.z);
  r.d2 = fmaf(r.dx, r.dx, fmaf(r.dy, r.dy, r.dz * r.dz));
  return r;
}

// One atom's pair sums, reduced over its T lanes (v: virial xx yy zz xy xz yz).
struct PairSums {
  float f[3], e, v[6];
};

template <int T, int V, bool EV, bool MULTI, class Fetch>
__device__ __forceinline__ PairSums lj_atom(const PairArgs& A, const LJF& P, const LJTabSmem& tab, int ntypes,
                                            double rcmax2, int64_t i, int lane, bool live, const Fetch& fetch) {
  // ROW: the cutoffs of a row's entries first, with one branch for the (rare)
  // entries in the band, where a branch an entry issues four times as many
  // instructions: 1M-atom LJ 144 -> 129 us, with energies 217 -> 183; 1M-atom
  // mixture with energies 315 -> 269.  A mixture without energies keeps the
  // branch an entry: at 64 registers a row's pairs spill 76 bytes (252 against
  // 227 us), and at 80 three blocks instead of four fit (264).
  constexpr bool ROW = !MULTI || EV;
  const int nn = live ? min(A.nnb[i], A.maxnb) : 0;
  const float4 pi = live ? A.posf[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  const int ti = __float_as_int(pi.w);
  float fx = 0.f, fy = 0.f, fz = 0.f, cfx = 0.f, cfy = 0.f, cfz = 0.f, e = 0.f, ce = 0.f;
  float v[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const ListRows<T, V> L(A.nbr, i, lane, A.stride, nn);
  for_rows(L, [&](const auto& R) {
    constexpr int N = sizeof(R.e) / sizeof(R.e[0]);
    float4 pj[N];
#pragma unroll
    for (int q = 0; q < N; ++q) pj[q] = fetch(R.e[q], R.e[q] & GBMD_IDX_MASK);
    float rx = 0.f, ry = 0.f, rz = 0.f, re = 0.f;
    auto term = [&](const GeomF& G, float sig2, float eps24, float eps4, float ecut, bool in) {
      // hardware reciprocal (within 1 ulp): the pair term's error budget is
      // ~1e-7 relative against a 1e-5 force tolerance
      float r2i;
      asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r2i) : "f"(G.d2));
      const float s2 = sig2 * r2i;
      const float s6 = s2 * s2 * s2;
      const float s12 = s6 * s6;
      const float fpair = in ? eps24 * fmaf(2.f, s12, -s6) * r2i : 0.f;  // -(dE/dr)/r
      rx = fmaf(-fpair, G.dx, rx);
      ry = fmaf(-fpair, G.dy, ry);
      rz = fmaf(-fpair, G.dz, rz);
      if (EV) {
        re += in ? 0.5f * fmaf(eps4, s12 - s6, -ecut) : 0.f;
        const float h = 0.5f * fpair;
        v[0] = fmaf(h * G.dx, G.dx, v[0]);
        v[1] = fmaf(h * G.dy, G.dy, v[1]);
        v[2] = fmaf(h * G.dz, G.dz, v[2]);
        v[3] = fmaf(h * G.dx, G.dy, v[3]);
        v[4] = fmaf(h * G.dx, G.dz, v[4]);
        v[5] = fmaf(h * G.dy, G.dz, v[5]);
      }
    };
    if constexpr (ROW) {
      GeomF Gs[N];
      int pids[N];
      bool ins[N], near = false;
#pragma unroll
      for (int q = 0; q < N; ++q) {
        Gs[q] = geom_f(R.e[q], pj[q], pi, A.g);
        pids[q] = MULTI ? ti * ntypes + __float_as_int(pj[q].w) : 0;
        const float2 lim = MULTI ? tab.b[pids[q]] : make_float2(P.rc2lo, P.rc2hi);
        ins[q] = Gs[q].d2 < lim.x;
        near |= !ins[q] && Gs[q].d2 <= lim.y;
      }
      if (near) {
#pragma unroll
        for (int q = 0; q < N; ++q)
          if (!ins[q] && Gs[q].d2 <= (MULTI ? tab.b[pids[q]].y : P.rc2hi) && R.ok[q])
            ins[q] = exact_inside(A.posd, i, R.e[q] & GBMD_IDX_MASK, R.e[q] >> GBMD_IDX_BITS, A.cellpack[i], A.g,
                                  MULTI ? rcmax2 : P.rc2, MULTI ? tab.r[pids[q]] : 0.0);
      }
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const float4 a = MULTI ? tab.a[pids[q]] : make_float4(P.sig2, P.eps24, P.eps4, P.ecut);
        term(Gs[q], a.x, a.y, a.z, a.w, ins[q]);
      }
    } else {
      // a mixture without energies; term's text again, since a call of it here
      // costs 8 % (244 against 227 us)
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const GeomF G = geom_u(R.e[q], pj[q], pi, A.g);
        int pid = ti * ntypes + __float_as_int(pj[q].w);
        const float4 a = tab.a[pid];
        const float2 b = tab.b[pid];
        // assigned, not initialised: the compiler then spills 8 bytes less (16.6 M
        // atoms, 20 steps: 106 against 114 ms)
        float sig2, eps24, rlo, rhi;
        sig2 = a.x;
        eps24 = a.y;
        rlo = b.x;
        rhi = b.y;
        bool in = G.d2 < rlo;
        if (!in && G.d2 <= rhi && R.ok[q])  // rare: the FP64 per-pair cutoff only here
          in = exact_inside(A.posd, i, R.e[q] & GBMD_IDX_MASK, R.e[q] >> GBMD_IDX_BITS, A.cellpack[i], A.g,
                            rcmax2, tab.r[pid]);
        float r2i;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r2i) : "f"(G.d2));
        const float s2 = sig2 * r2i;
        const float s6 = s2 * s2 * s2;
        const float s12 = s6 * s6;
        const float fpair = in ? eps24 * fmaf(2.f, s12, -s6) * r2i : 0.f;  // -(dE/dr)/r
        rx = fmaf(-fpair, G.dx, rx);
        ry = fmaf(-fpair, G.dy, ry);
        rz = fmaf(-fpair, G.dz, rz);
      }
    }
    kahan_add(fx, cfx, rx);
    kahan_add(fy, cfy, ry);
    kahan_add(fz, cfz, rz);
    if (EV) kahan_add(e, ce, re);
  });
  group_reduce_kahan<T>(fx, cfx);
  group_reduce_kahan<T>(fy, cfy);
  group_reduce_kahan<T>(fz, cfz);
  PairSums S;
  S.f[0] = fx - cfx;
  S.f[1] = fy - cfy;
  S.f[2] = fz - cfz;
  S.e = 0.f;
  if (EV) {
    group_reduce_kahan<T>(e, ce);
    reduce6(v, T);
    S.e = e - ce;
#pragma unroll
    for (int q = 0; q < 6; ++q) S.v[q] = v[q];
  }
  return S;
}

// Epilogue of one atom from its pair sums; emb: its embedding energy.  The
// virial row is written here too, 72 bytes apart from lane to lane: for the
// kernels whose blocks have no common loop (block_epilogue is the other).
template <bool EV>
__device__ __forceinline__ void atom_finish(const PairArgs& A, int64_t i, const PairSums& S, float emb) {
  const int ti = __float_as_int(A.posf[i].w);
  const float im = A.inv_massf[ti];
  double o[9];
  if (EV) vir9(S.v, o);
  atom_epilogue<true>(A, i, ti, 0., 0., 0., S.f[0] * im, S.f[1] * im, S.f[2] * im,
                      EV ? (double)emb + (double)S.e : 0.0, EV ? o : nullptr);
}

// Epilogue of a block's atoms i0 .. i0 + blockDim / T, whose sums the groups'
// first lanes hold.  They pass through shared memory to the block's first
// blockDim / T threads, so that the per-atom work (the FP64 Verlet halves,
// the stores) runs on full warps: on each group's first lane alone it would
// issue T times as many FP64 instructions, 16 SM cycles each.  The virial rows (9 doubles per atom) go through shared
// memory so that the block writes them contiguously; a lane writing its own
// row touches 32 sectors per store, nine times.
template <int T, bool EV>
__device__ __forceinline__ void block_epilogue(const PairArgs& A, int64_t i0, const PairSums& S,
                                               const float* __restrict__ epf) {
  constexpr int NV = EV ? 10 : 3;
  constexpr bool SHARED = T > 1 || EV;
  __shared__ float sums[SHARED ? NV : 1][SHARED ? 256 / T : 1];
  const int nat = (int)blockDim.x / T;
  PairSums R = S;
  if (SHARED) {
    const int a = (int)threadIdx.x / T;
    if (threadIdx.x % T == 0) {
#pragma unroll
      for (int q = 0; q < 3; ++q) sums[q][a] = S.f[q];
      if (EV) {
        sums[3][a] = S.e;
#pragma unroll
        for (int q = 0; q < 6; ++q) sums[4 + q][a] = S.v[q];
      }
    }
    __syncwarp();  // the lanes' lists differ in length
    __syncthreads();
    if (EV && A.want_virial) {
      const int m = (int)min((int64_t)nat, A.n - i0) * 9;
      for (int k = threadIdx.x; k < m; k += blockDim.x) {
        const int q = k % 9;  // row-major 3x3 from xx yy zz xy xz yz
        A.vir[9 * i0 + k] = widen(sums[4 + ((0x254513430u >> (4 * q)) & 15)][k / 9]);
      }
    }
    if ((int)threadIdx.x >= nat) return;
    if (T > 1) {
#pragma unroll
      for (int q = 0; q < 3; ++q) R.f[q] = sums[q][threadIdx.x];
      if (EV) R.e = sums[3][threadIdx.x];
    }
  }
  const int64_t i = i0 + threadIdx.x;
  if (i >= A.n) return;
  const int ti = __float_as_int(A.posf[i].w);
  const float im = A.inv_massf[ti];
  atom_epilogue<true>(A, i, ti, 0., 0., 0., R.f[0] * im, R.f[1] * im, R.f[2] * im,
                      EV ? (epf ? (double)epf[i] : 0.0) + (double)R.e : 0.0, nullptr);
}

// PIECE: the launch covers atoms [A.i0, A.n) only (a separate instantiation:
// the offset costs registers that the full-range kernel, at the 64-register
// cap, would spill).
template <int T, int V, bool EV, bool MULTI, bool PIECE>
__global__ void __launch_bounds__(256, EV ? 3 : 4) k_lj_mixed(PairArgs A, LJF P, const LJPair* __restrict__ tab, int ntypes,
                                                  double rcmax2) {
  __shared__ LJTabSmem t;
  if (MULTI) lj_load_table(t, tab, ntypes);
  const int64_t gt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t i = PIECE ? A.i0 + gt / T : gt / T;
  const PairSums S =
      lj_atom<T, V, EV, MULTI>(A, P, t, ntypes, rcmax2, i, (int)(gt % T), i < A.n, GlobalFetch{A.posf});
  block_epilogue<T, EV>(A, (PIECE ? A.i0 : 0) + blockIdx.x * (int64_t)(blockDim.x / T), S, nullptr);
}

// One lane per atom, 4 entries per load, neighbour positions from the
// block's staged cells.
template <bool EV, bool MULTI>
__global__ void __launch_bounds__(256) k_lj_staged(PairArgs A, LJF P, const LJPair* __restrict__ tab, int ntypes,
                                                   double rcmax2, const int32_t* __restrict__ cstart, int K,
                                                   int cap) {
  __shared__ LJTabSmem t;
  __shared__ int4 rows[16];
  __shared__ int sh[56];
  extern __shared__ float4 staged_pos[];
  if (MULTI) lj_load_table(t, tab, ntypes);
  int64_t a0, a1;
  const bool ok = stage_cells(A.g, cstart, A.posf, K, cap, staged_pos, rows, sh, a0, a1);
  for (int64_t i = a0 + threadIdx.x; i < a1; i += blockDim.x) {
    const PairSums S = ok ? lj_atom<1, 4, EV, MULTI>(A, P, t, ntypes, rcmax2, i, 0, true, StagedFetch{staged_pos, rows})
                          : lj_atom<1, 4, EV, MULTI>(A, P, t, ntypes, rcmax2, i, 0, true, GlobalFetch{A.posf});
    atom_finish<EV>(A, i, S, 0.f);
  }
}

// ---------------------------------------------------------------------------
// eam_alloy
// ---------------------------------------------------------------------------
__device__ __forceinline__ int knot_f(float r, float rdr, int nr, float& q) {
  float t = fmaf(r, rdr, 1.0f);
  const int m = min((int)t, nr - 1);
  q = fminf(t - (float)m, 1.0f);
  return m;
}

__device__ __forceinline__ float spline_val(const float4& c, float q) {
  return fmaf(fmaf(fmaf(c.x, q, c.y), q, c.z), q, c.w);
}

__device__ __forceinline__ float spline_der(const float4& c, float q, float rd) {
  return fmaf(fmaf(3.f * c.x, q, 2.f * c.y), q, c.z) * rd;
}

// Density of atom i, reduced over its T lanes.
template <int T, int V, bool SINGLE, class Fetch>
__device__ __forceinline__ float eam_rho_atom(const PairArgs& A, const EamDev& E, int64_t i, int lane, bool live,
                                              const Fetch& fetch) {
  const int nn = live ? min(A.nnb[i], A.maxnb) : 0;
  const float4 pi = live ? A.posf[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  const int nr = E.nr, nr1 = E.nr + 1;
  const float rdr = E.rdrf;
  float rho = 0.f, crho = 0.f;
  const PairFrame PF(pi, A.g);
  const ListRows<T, V> L(A.nbr, i, lane, A.stride, nn);
  for_rows(L, [&](const auto& R) {
    constexpr int N = sizeof(R.e) / sizeof(R.e[0]);
    float4 pj[N];
#pragma unroll
    for (int q = 0; q < N; ++q) pj[q] = fetch(R.e[q], R.e[q] & GBMD_IDX_MASK);
    auto retest = [&](int q) {
      return exact_inside(A.posd, i, R.e[q] & GBMD_IDX_MASK, R.e[q] >> GBMD_IDX_BITS, A.cellpack[i], A.g, E.rcut2,
                          0.0);
    };
    float rr = 0.f;
    if constexpr (N % 2 == 0) {
      // entries (0, 1) and (2, 3) in packed FP32; the rows' partial sums
      // stay packed until the row is added to the compensated sum
      float2 rr2 = f2(0.f, 0.f);
#pragma unroll
      for (int q = 0; q < N; q += 2) {
        const GeomF2 G = PF.geom(R.e[q], R.e[q + 1], pj[q], pj[q + 1]);
        bool ina = G.d2.x < E.rc2lo, inb = G.d2.y < E.rc2lo;
        if (!ina && G.d2.x <= E.rc2hi && R.ok[q]) ina = retest(q);
        if (!inb && G.d2.y <= E.rc2hi && R.ok[q + 1]) inb = retest(q + 1);
        const float2 rd = __fmul2_rn(G.d2, f2(rsqrtf(G.d2.x), rsqrtf(G.d2.y)));
        const float2 tt = __ffma2_rn(rd, f2(rdr, rdr), f2(1.0f, 1.0f));
        const int ma = min((int)tt.x, nr - 1), mb = min((int)tt.y, nr - 1);
        const float2 qq0 = __fadd2_rn(tt, f2(-(float)ma, -(float)mb));
        const float2 qq = f2(fminf(qq0.x, 1.0f), fminf(qq0.y, 1.0f));
        const float4 ca = __ldg(&E.rhor4[SINGLE ? ma : __float_as_int(pj[q].w) * nr1 + ma]);
        const float4 cb = __ldg(&E.rhor4[SINGLE ? mb : __float_as_int(pj[q + 1].w) * nr1 + mb]);
        const float2 val = __ffma2_rn(__ffma2_rn(__ffma2_rn(f2(ca.x, cb.x), qq, f2(ca.y, cb.y)), qq, f2(ca.z, cb.z)),
                                      qq, f2(ca.w, cb.w));
        rr2 = __fadd2_rn(rr2, f2(ina ? val.x : 0.f, inb ? val.y : 0.f));
      }
      rr = rr2.x + rr2.y;
    } else {
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const GeomF G = geom_f(R.e[q], pj[q], pi, A.g);
        bool in = G.d2 < E.rc2lo;
        if (!in && G.d2 <= E.rc2hi && R.ok[q]) in = retest(q);
        const float rd = G.d2 * rsqrtf(G.d2);
        float t;
        const int m = knot_f(rd, rdr, nr, t);
        const float4 c = __ldg(&E.rhor4[SINGLE ? m : __float_as_int(pj[q].w) * nr1 + m]);
        rr += in ? spline_val(c, t) : 0.f;
      }
    }
    kahan_add(rho, crho, rr);
  });
  group_reduce_kahan<T>(rho, crho);
  return rho - crho;
}

// Rho2EmbOp / eam_alloy_fEmbed of one atom: F'(rho) (and F(rho) on energy
// steps), linear continuation above rhomax.  SINGLE (one element): also
// writes pfp[i] = (position, F'(rho_i)) so the force pass gathers both in one
// 16 B load.
template <bool EV, bool SINGLE>
__device__ __forceinline__ float eam_embed(const PairArgs& A, const EamDev& E, int64_t i, float R,
                                          float* __restrict__ fpf, float* __restrict__ epf,
                                          float4* __restrict__ pfp) {
  const float4 pi = A.posf[i];
  const int ti = SINGLE ? 0 : __float_as_int(pi.w);
  float q = fmaf(R, E.rdrhof, 1.0f);
  int m = (int)q;
  m = max(1, min(m, E.nrho - 1));
  q = fminf(q - (float)m, 1.0f);
  const float4 c = __ldg(&E.frho4[(SINGLE ? 0 : ti * (E.nrho + 1)) + m]);
  const float fp = spline_der(c, q, E.rdrhof);
  fpf[i] = fp;
  if (SINGLE) pfp[i] = make_float4(pi.x, pi.y, pi.z, fp);
  if (EV) {
    float phi = spline_val(c, q);
    if (R > E.rhomaxf) phi = fmaf(fp, R - E.rhomaxf, phi);
    epf[i] = phi;
  }
  return fp;
}

template <int T, int V, bool EV, bool SINGLE, bool PIECE>
__global__ void __launch_bounds__(256) k_eam_rho_mixed(PairArgs A, EamDev E, float* __restrict__ fpf,
                                                       float* __restrict__ epf, float4* __restrict__ pfp) {
  const int64_t gt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int64_t i = PIECE ? A.i0 + gt / T : gt / T;
  float R = eam_rho_atom<T, V, SINGLE>(A, E, i, (int)(gt % T), i < A.n, GlobalFetch{A.posf});
  if (T > 1) {
    // the embedding of the block's atoms on its first blockDim / T threads
    __shared__ float rho[T > 1 ? 256 / T : 1];
    const int nat = (int)blockDim.x / T;
    if (threadIdx.x % T == 0) rho[threadIdx.x / T] = R;
    __syncwarp();
    __syncthreads();
    if ((int)threadIdx.x >= nat) return;
    R = rho[threadIdx.x];
    i = (PIECE ? A.i0 : 0) + blockIdx.x * (int64_t)nat + threadIdx.x;
  }
  if (i < A.n) eam_embed<EV, SINGLE>(A, E, i, R, fpf, epf, pfp);
}

template <bool EV>
__global__ void __launch_bounds__(256) k_eam_rho_staged(PairArgs A, EamDev E, float* __restrict__ fpf,
                                                        float* __restrict__ epf, float4* __restrict__ pfp,
                                                        const int32_t* __restrict__ cstart, int K, int cap) {
  __shared__ int4 rows[16];
  __shared__ int sh[56];
  extern __shared__ float4 staged_pos[];
  int64_t a0, a1;
  const bool ok = stage_cells(A.g, cstart, A.posf, K, cap, staged_pos, rows, sh, a0, a1);
  for (int64_t i = a0 + threadIdx.x; i < a1; i += blockDim.x) {
    const float R = ok ? eam_rho_atom<1, 4, true>(A, E, i, 0, true, StagedFetch{staged_pos, rows})
                       : eam_rho_atom<1, 4, true>(A, E, i, 0, true, GlobalFetch{A.posf});
    eam_embed<EV, true>(A, E, i, R, fpf, epf, pfp);
  }
}

// One 32-byte load of a knot's two float4 (rho' and z2r coefficients of the
// interleaved one-element table; the address is 32-byte aligned).
__device__ __forceinline__ void ldg_knot_pair(const float4* p, float4& a, float4& b) {
  asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(p));
}

__device__ __forceinline__ int z2r_index_d(int a, int b) {
  const int irow = a > b ? a : b, icol = a > b ? b : a;
  return irow * (irow + 1) / 2 + icol;
}

// Force pass: f_i = sum_j u_ij (F'_i rho_j'(r) + F'_j rho_i'(r) + phi'(r)).
// SINGLE reads (position, F'_j) through `fetch` from pfp; otherwise position
// (type in w) and fpf.
template <int T, int V, bool EV, bool SINGLE, class Fetch>
__device__ __forceinline__ PairSums eam_force_atom(const PairArgs& A, const EamDev& E, const float* __restrict__ fpf,
                                                   int64_t i, int lane, bool live, const Fetch& fetch) {
  const int nn = live ? min(A.nnb[i], A.maxnb) : 0;
  const float4 pi = live ? A.posf[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  const float fpi = live ? fpf[i] : 0.f;
  const int ti = SINGLE ? 0 : __float_as_int(pi.w);
  const int nr = E.nr, nr1 = E.nr + 1;
  const float rdr = E.rdrf;
  float fx = 0.f, fy = 0.f, fz = 0.f, cfx = 0.f, cfy = 0.f, cfz = 0.f, e = 0.f, ce = 0.f;
  float v[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const ListRows<T, V> L(A.nbr, i, lane, A.stride, nn);
  for_rows(L, [&](const auto& R) {
    constexpr int N = sizeof(R.e) / sizeof(R.e[0]);
    float4 pj[N];
    float fpj[N];
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const uint32_t j = R.e[q] & GBMD_IDX_MASK;
      pj[q] = fetch(R.e[q], j);
      fpj[q] = SINGLE ? pj[q].w : __ldg(&fpf[j]);
    }
    float rx = 0.f, ry = 0.f, rz = 0.f, re = 0.f;
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const GeomF G = geom_f(R.e[q], pj[q], pi, A.g);
      bool in = G.d2 < E.rc2lo;
      if (!in && G.d2 <= E.rc2hi && R.ok[q])
        in = exact_inside(A.posd, i, R.e[q] & GBMD_IDX_MASK, R.e[q] >> GBMD_IDX_BITS, A.cellpack[i], A.g, E.rcut2,
                          0.0);
      const float rs = rsqrtf(G.d2);
      const float rd = G.d2 * rs;
      float t;
      const int m = knot_f(rd, rdr, nr, t);
      const int tj = SINGLE ? 0 : __float_as_int(pj[q].w);
      // rho'(r) from the pre-scaled derivative table: (3c3/dr, 2c4/dr, c5/dr);
      // one element: rho' and z2r knots interleaved, read in one 32 B load
      float4 dj, cz;
      if (SINGLE) {
        ldg_knot_pair(&E.fz8[2 * m], dj, cz);
      } else {
        dj = __ldg(&E.rhod4[tj * nr1 + m]);
        cz = __ldg(&E.z2r4[z2r_index_d(ti, tj) * nr1 + m]);
      }
      const float rhojp = fmaf(fmaf(dj.x, t, dj.y), t, dj.z);
      float rhoip = rhojp;
      if (!SINGLE && ti != tj) {
        const float4 di = __ldg(&E.rhod4[ti * nr1 + m]);
        rhoip = fmaf(fmaf(di.x, t, di.y), t, di.z);
      }
      const float t1 = fmaf(cz.x, t, cz.y);
      const float z2 = fmaf(fmaf(t1, t, cz.z), t, cz.w);          // z2r tables carry conv_z2r
      const float z2d = fmaf(fmaf(cz.x, t, t1 + t1), t, cz.z);     // d z2 / d t
      const float phi = z2 * rs;
      const float phip = fmaf(z2d * rdr, rs, -phi * rs);
      const float psip = fmaf(fpi, rhojp, fmaf(fpj[q], rhoip, phip));
      const float fpair = in ? psip * rs : 0.f;
      rx = fmaf(G.dx, fpair, rx);
      ry = fmaf(G.dy, fpair, ry);
      rz = fmaf(G.dz, fpair, rz);
      if (EV) {
        re += in ? 0.5f * phi : 0.f;
        const float h = -0.5f * fpair;
        v[0] = fmaf(h * G.dx, G.dx, v[0]);
        v[1] = fmaf(h * G.dy, G.dy, v[1]);
        v[2] = fmaf(h * G.dz, G.dz, v[2]);
        v[3] = fmaf(h * G.dx, G.dy, v[3]);
        v[4] = fmaf(h * G.dx, G.dz, v[4]);
        v[5] = fmaf(h * G.dy, G.dz, v[5]);
      }
    }
    kahan_add(fx, cfx, rx);
    kahan_add(fy, cfy, ry);
    kahan_add(fz, cfz, rz);
    if (EV) kahan_add(e, ce, re);
  });
  group_reduce_kahan<T>(fx, cfx);
  group_reduce_kahan<T>(fy, cfy);
  group_reduce_kahan<T>(fz, cfz);
  PairSums S;
  S.f[0] = fx - cfx;
  S.f[1] = fy - cfy;
  S.f[2] = fz - cfz;
  S.e = 0.f;
  if (EV) {
    group_reduce_kahan<T>(e, ce);
    reduce6(v, T);
    S.e = e - ce;
#pragma unroll
    for (int q = 0; q < 6; ++q) S.v[q] = v[q];
  }
  return S;
}

template <int T, int V, bool EV, bool SINGLE, bool PIECE>
__global__ void __launch_bounds__(256, EV ? 3 : 4) k_eam_force_mixed(PairArgs A, EamDev E, const float* __restrict__ fpf,
                                                         const float* __restrict__ epf,
                                                         const float4* __restrict__ pfp) {
  const int64_t gt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t i = PIECE ? A.i0 + gt / T : gt / T;
  const PairSums S = eam_force_atom<T, V, EV, SINGLE>(A, E, fpf, i, (int)(gt % T), i < A.n,
                                                      GlobalFetch{SINGLE ? pfp : A.posf});
  block_epilogue<T, EV>(A, (PIECE ? A.i0 : 0) + blockIdx.x * (int64_t)(blockDim.x / T), S, epf);
}

template <bool EV>
__global__ void __launch_bounds__(256) k_eam_force_staged(PairArgs A, EamDev E, const float* __restrict__ fpf,
                                                          const float* __restrict__ epf,
                                                          const float4* __restrict__ pfp,
                                                          const int32_t* __restrict__ cstart, int K, int cap) {
  __shared__ int4 rows[16];
  __shared__ int sh[56];
  extern __shared__ float4 staged_pos[];
  int64_t a0, a1;
  const bool ok = stage_cells(A.g, cstart, pfp, K, cap, staged_pos, rows, sh, a0, a1);
  for (int64_t i = a0 + threadIdx.x; i < a1; i += blockDim.x) {
    const PairSums S = ok ? eam_force_atom<1, 4, EV, true>(A, E, fpf, i, 0, true, StagedFetch{staged_pos, rows})
                          : eam_force_atom<1, 4, EV, true>(A, E, fpf, i, 0, true, GlobalFetch{pfp});
    atom_finish<EV>(A, i, S, EV ? epf[i] : 0.f);
  }
}

// ---------------------------------------------------------------------------
// One-element eam_alloy forces without energies.  The force on i is
//   sum_j phi'(r) u + sum_j (F'_i + F'_j) rho'(r) u.
// The density pass has every pair's knot at hand, so it forms the first sum
// (f0) too and leaves rho'(r) / r for each list entry in `bpair`, laid out as
// the list.  The force pass is left with the second: per entry 4 + 4 streamed
// bytes, one 16 B gather and some 25 instructions, where the pair terms' own
// knots (32 B a lane, 28 lines a warp) made it the larger of the two.  The
// streamed floats go through HBM, which both passes left at a fifth of its
// rate; they bypass L1, which serves the gathers.
// 4 M-atom Cu, density + force: 529 + 768 -> 796 + 411 us (72 registers in the
// density pass; 64: 810, 56: 972).
// (Two elements: the entry's two rho' differ, and the sum over F'_i has to be
// formed in the density pass as well; that was slower than the plain passes,
// 2 M atoms 933 against 874 us.)
// ---------------------------------------------------------------------------
struct BondSums {
  float rho, s[3], c[3];  // force sum s - c, unrounded
};

// f0 keeps both parts, so that the force is rounded once, as one compensated sum
// over both passes would be: f, and in w the three low parts, 10 bits each, in
// units of 2^-9 of the last place of f (below half of which they lie), to and
// from integers through the mantissa.
__device__ __forceinline__ int low_part(float f, float lo) {
  const float to = __int_as_float(0x7f000000 - (__float_as_int(f) & 0x7f800000));  // 1 / the power of two below f
  return __float_as_int(fmaf(lo * to, 0x1p32f, 12582912.0f)) & 1023;
}
__device__ __forceinline__ float low_part_of(float f, int bits) {
  const float q = __int_as_float(0x4b000000 | ((bits & 1023) ^ 512)) - 8389120.0f;
  return __int_as_float(__float_as_int(f) & 0x7f800000) * (q * 0x1p-32f);
}
__device__ __forceinline__ float4 pack_f0(const BondSums& S) {
  float f[3];
  int w = 0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    f[k] = S.s[k] - S.c[k];
    w |= low_part(f[k], (S.s[k] - f[k]) - S.c[k]) << (10 * k);
  }
  return make_float4(f[0], f[1], f[2], __int_as_float(w));
}

// (a + alo) + (b + blo), rounded once but for the low parts' own rounding.
__device__ __forceinline__ float sum_parts(float a, float alo, float b, float blo) {
  const float t = a + b, z = t - a, e = (a - (t - z)) + (b - z);
  return t + (e + (alo + blo));
}

// The force sum of both passes from the force pass's.
__device__ __forceinline__ void add_f0(const PairArgs& A, int64_t i, const BondSums& S, float (&f)[3]) {
  const float4 a = __ldg(&A.f0[i]);
  const int w = __float_as_int(a.w);
  f[0] = sum_parts(a.x, low_part_of(a.x, w), S.s[0], -S.c[0]);
  f[1] = sum_parts(a.y, low_part_of(a.y, w >> 10), S.s[1], -S.c[1]);
  f[2] = sum_parts(a.z, low_part_of(a.z, w >> 20), S.s[2], -S.c[2]);
}

template <int T, class Fetch>
__device__ __forceinline__ BondSums eam_rho_bonds_atom(const PairArgs& A, const EamDev& E, int64_t i, int lane,
                                                       bool live, const Fetch& fetch) {
  const int nn = live ? min(A.nnb[i], A.maxnb) : 0;
  const float4 pi = live ? A.posf[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  const int nr = E.nr;
  const float rdr = E.rdrf;
  float s[4], c[4];  // rho, sum phi'/r d
#pragma unroll
  for (int k = 0; k < 4; ++k) s[k] = c[k] = 0.f;
  const ListRows<T, 4> L(A.nbr, i, lane, A.stride, nn);
  float* const bonds = A.bpair + (L.p - A.nbr);
  for_rows(L, [&](const auto& R) {
    constexpr int N = sizeof(R.e) / sizeof(R.e[0]);
    float4 pj[N];
#pragma unroll
    for (int q = 0; q < N; ++q) pj[q] = fetch(R.e[q], R.e[q] & GBMD_IDX_MASK);
    float p[4], b[N];
#pragma unroll
    for (int k = 0; k < 4; ++k) p[k] = 0.f;
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const GeomF G = geom_u(R.e[q], pj[q], pi, A.g);
      bool in = G.d2 < E.rc2lo;
      if (!in && G.d2 <= E.rc2hi && R.ok[q])
        in = exact_inside(A.posd, i, R.e[q] & GBMD_IDX_MASK, R.e[q] >> GBMD_IDX_BITS, A.cellpack[i], A.g, E.rcut2,
                          0.0);
      const float rs = rsqrtf(G.d2);
      const float rd = G.d2 * rs;
      float t;
      const int m = knot_f(rd, rdr, nr, t);
      float4 cr, cz;
      ldg_knot_pair(&E.rz8[2 * m], cr, cz);
      const float t1 = fmaf(cz.x, t, cz.y);
      const float z2 = fmaf(fmaf(t1, t, cz.z), t, cz.w);
      const float z2d = fmaf(fmaf(cz.x, t, t1 + t1), t, cz.z);
      const float phi = z2 * rs;
      const float phip = fmaf(z2d * rdr, rs, -phi * rs);
      const float fa = in ? phip * rs : 0.f;
      b[q] = in ? spline_der(cr, t, rdr) * rs : 0.f;
      p[0] += in ? spline_val(cr, t) : 0.f;
      p[1] = fmaf(G.dx, fa, p[1]);
      p[2] = fmaf(G.dy, fa, p[2]);
      p[3] = fmaf(G.dz, fa, p[3]);
    }
    if constexpr (N == 4)
      asm volatile("st.global.L1::no_allocate.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(bonds + R.at), "f"(b[0]), "f"(b[1]),
                   "f"(b[2]), "f"(b[3])
                   : "memory");
    else
      *reinterpret_cast<float2*>(bonds + R.at) = make_float2(b[0], b[1]);
#pragma unroll
    for (int k = 0; k < 4; ++k) kahan_add(s[k], c[k], p[k]);
  });
#pragma unroll
  for (int k = 0; k < 4; ++k) group_reduce_kahan<T>(s[k], c[k]);
  return BondSums{s[0] - c[0], {s[1], s[2], s[3]}, {c[1], c[2], c[3]}};
}

template <int T, bool PIECE>
__global__ void __launch_bounds__(128, 7) k_eam_rho_bonds(const __grid_constant__ PairArgs A,
                                                          const __grid_constant__ EamDev E,
                                                          float* __restrict__ fpf, float4* __restrict__ pfp) {
  const int64_t gt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int64_t i = PIECE ? A.i0 + gt / T : gt / T;
  const BondSums S = eam_rho_bonds_atom<T>(A, E, i, (int)(gt % T), i < A.n, GlobalFetch{A.posf});
  float rho = S.rho;
  float4 f0 = pack_f0(S);
  if (T > 1) {
    // the embedding of the block's atoms on its first blockDim / T threads.  Five
    // floats an atom: with seven (the sums unpacked) the seven blocks of an SM
    // take the next size of shared memory from L1 (864,000 atoms: 184 -> 192 us)
    __shared__ float sums[5][T > 1 ? 128 / T : 1];
    const int nat = (int)blockDim.x / T;
    if (threadIdx.x % T == 0) {
      const int a = (int)threadIdx.x / T;
      sums[0][a] = rho;
      sums[1][a] = f0.x;
      sums[2][a] = f0.y;
      sums[3][a] = f0.z;
      sums[4][a] = f0.w;
    }
    __syncwarp();
    __syncthreads();
    if ((int)threadIdx.x >= nat) return;
    rho = sums[0][threadIdx.x];
    f0 = make_float4(sums[1][threadIdx.x], sums[2][threadIdx.x], sums[3][threadIdx.x], sums[4][threadIdx.x]);
    i = (PIECE ? A.i0 : 0) + blockIdx.x * (int64_t)nat + threadIdx.x;
  }
  if (i >= A.n) return;
  A.f0[i] = f0;
  eam_embed<false, true>(A, E, i, rho, fpf, nullptr, pfp);
}

template <int T, class Fetch>
__device__ __forceinline__ BondSums eam_force_bonds_atom(const PairArgs& A, const float* __restrict__ fpf, int64_t i,
                                                         int lane, bool live, const Fetch& fetch) {
  const int nn = live ? min(A.nnb[i], A.maxnb) : 0;
  const float4 pi = live ? A.posf[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  const float fpi = live ? fpf[i] : 0.f;
  float s[3] = {0.f, 0.f, 0.f}, c[3] = {0.f, 0.f, 0.f};
  const ListRows<T, 4> L(A.nbr, i, lane, A.stride, nn);
  const float* const bonds = A.bpair + (L.p - A.nbr);
  auto load = [&](int r, uint32_t (&e)[4], float (&b)[4]) {
    L.load(r, e);
    asm("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];"
        : "=f"(b[0]), "=f"(b[1]), "=f"(b[2]), "=f"(b[3])
        : "l"(bonds + (size_t)r * L.stride));
  };
  uint32_t ent[4], nxt[4];
  float b[4], nb[4];
  if (L.nrow > 0) load(0, ent, b);
  for (int r = 0; r < L.nrow; ++r) {
    if (r + 1 < L.nrow) load(r + 1, nxt, nb);
    if (r >= L.nfull) {  // the last, partial row
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (!L.in_tail(q)) {
          ent[q] = L.standin;
          b[q] = 0.f;
        }
    }
    float4 pj[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) pj[q] = fetch(ent[q], ent[q] & GBMD_IDX_MASK);
    float p[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float w = (fpi + pj[q].w) * b[q];
      p[0] = fmaf(fmaf(unit_of(ent[q] >> 26), A.g.hf[0], pj[q].x - pi.x), w, p[0]);
      p[1] = fmaf(fmaf(unit_of(ent[q] >> 28), A.g.hf[1], pj[q].y - pi.y), w, p[1]);
      p[2] = fmaf(fmaf(unit_of(ent[q] >> 30), A.g.hf[2], pj[q].z - pi.z), w, p[2]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) kahan_add(s[k], c[k], p[k]);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      ent[q] = nxt[q];
      b[q] = nb[q];
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) group_reduce_kahan<T>(s[k], c[k]);
  return BondSums{0.f, {s[0], s[1], s[2]}, {c[0], c[1], c[2]}};
}

template <int T, bool PIECE>
__global__ void __launch_bounds__(256, 4) k_eam_force_bonds(const __grid_constant__ PairArgs A,
                                                            const float* __restrict__ fpf,
                                                            const float4* __restrict__ pfp) {
  const int64_t gt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int64_t i = PIECE ? A.i0 + gt / T : gt / T;
  BondSums S = eam_force_bonds_atom<T>(A, fpf, i, (int)(gt % T), i < A.n, GlobalFetch{pfp});
  // the epilogue of the block's atoms on its first blockDim / T threads, as block_epilogue's
  if (T > 1) {
    __shared__ float sums[6][T > 1 ? 256 / T : 1];
    const int nat = (int)blockDim.x / T;
    if (threadIdx.x % T == 0) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        sums[k][threadIdx.x / T] = S.s[k];
        sums[3 + k][threadIdx.x / T] = S.c[k];
      }
    }
    __syncwarp();
    __syncthreads();
    if ((int)threadIdx.x >= nat) return;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      S.s[k] = sums[k][threadIdx.x];
      S.c[k] = sums[3 + k][threadIdx.x];
    }
    i = (PIECE ? A.i0 : 0) + blockIdx.x * (int64_t)nat + threadIdx.x;
  }
  if (i >= A.n) return;
  float f[3];
  add_f0(A, i, S, f);
  const int ti = __float_as_int(A.posf[i].w);
  const float im = A.inv_massf[ti];
  atom_epilogue<true>(A, i, ti, 0., 0., 0., f[0] * im, f[1] * im, f[2] * im, 0.0, nullptr);
}

// The same with the neighbour positions from the block's staged cells.
__global__ void __launch_bounds__(256) k_eam_rho_bonds_staged(const __grid_constant__ PairArgs A,
                                                              const __grid_constant__ EamDev E,
                                                              float* __restrict__ fpf, float4* __restrict__ pfp,
                                                              const int32_t* __restrict__ cstart, int K, int cap) {
  __shared__ int4 rows[16];
  __shared__ int sh[56];
  extern __shared__ float4 staged_pos[];
  int64_t a0, a1;
  const bool ok = stage_cells(A.g, cstart, A.posf, K, cap, staged_pos, rows, sh, a0, a1);
  for (int64_t i = a0 + threadIdx.x; i < a1; i += blockDim.x) {
    const BondSums S = ok ? eam_rho_bonds_atom<1>(A, E, i, 0, true, StagedFetch{staged_pos, rows})
                          : eam_rho_bonds_atom<1>(A, E, i, 0, true, GlobalFetch{A.posf});
    eam_embed<false, true>(A, E, i, S.rho, fpf, nullptr, pfp);
    A.f0[i] = pack_f0(S);
  }
}

__global__ void __launch_bounds__(256) k_eam_force_bonds_staged(const __grid_constant__ PairArgs A,
                                                                const float* __restrict__ fpf,
                                                                const float4* __restrict__ pfp,
                                                                const int32_t* __restrict__ cstart, int K, int cap) {
  __shared__ int4 rows[16];
  __shared__ int sh[56];
  extern __shared__ float4 staged_pos[];
  int64_t a0, a1;
  const bool ok = stage_cells(A.g, cstart, pfp, K, cap, staged_pos, rows, sh, a0, a1);
  for (int64_t i = a0 + threadIdx.x; i < a1; i += blockDim.x) {
    const BondSums B = ok ? eam_force_bonds_atom<1>(A, fpf, i, 0, true, StagedFetch{staged_pos, rows})
                          : eam_force_bonds_atom<1>(A, fpf, i, 0, true, GlobalFetch{pfp});
    PairSums S;
    add_f0(A, i, B, S.f);
    S.e = 0.f;
    atom_finish<false>(A, i, S, 0.f);
  }
}

// ---------------------------------------------------------------------------
// Newton-3 LJ (lj_compute_force_symetric, pair_potential_singlemat_symetric.cpp
// L230-320): every unordered pair once, from the half list (j after i in cell
// order).  The pair's force, half its energy and half its virial go to i's
// register sums and -- the force negated -- to j's accumulators (the
// reference takes a spin lock on j); i's own sums are added to its
// accumulators once at the end, since other threads add to them as well.
//
// The accumulators are 64-bit fixed-point integers, so the sums do not depend
// on the order the additions arrive in and the results are the same from run
// to run.  Ten planes of `cap`: f (3), ep, virial xx yy zz xy xz yz.  A value
// x is stored as round(x * 2^38 / b), b a power of two bounding its kind (24
// eps/sigma for forces, 4 eps for energies, that force times rcut for
// virials): x * 2^38 / b is exact in FP32 and the rounding is deterministic.
// A pair's contribution must stay below 2^16 b, i's own sum below 2^24 b, so
// that 512 of them cannot overflow 2^63; a larger one raises
// GBMD_DEVERR_RANGE.  k_h3_epilogue turns the sums into the acceleration
// (and the fused Verlet half steps) and clears them for the next pass.
// ---------------------------------------------------------------------------
struct FixScale {
  float f, e, v, r;    // 2^38 / bound for forces, energies, virials, EAM densities
  double inv_f, inv_e, inv_v, inv_r;
  int* err;
};

constexpr float FIX_PAIR_LIMIT = 0x1p54f;  // |x * scale| of one pair's contribution
constexpr float FIX_SUM_LIMIT = 0x1p62f;   // |x * scale| of an atom's own sum

__device__ __forceinline__ long long fix_q(float x, float scale, float limit, int* err) {
  float y = x * scale;
  if (!(fabsf(y) <= limit)) {
    atomicOr(err, GBMD_DEVERR_RANGE);
    y = y != y ? 0.f : copysignf(limit, y);
  }
  return __float2ll_rn(y);
}

__device__ __forceinline__ void fix_add(long long* p, long long q) {
  // two's complement: the unsigned sum is the signed one modulo 2^64
  atomicAdd(reinterpret_cast<unsigned long long*>(p), (unsigned long long)q);
}

template <bool EV, bool MULTI>
__global__ void __launch_bounds__(256, EV ? 1 : 4) k_lj_half(PairArgs A, LJF P, const LJPair* __restrict__ tab, int ntypes,
                                                 double rcmax2, long long* __restrict__ acc, int64_t cap,
                                                 FixScale X) {
  __shared__ LJTabSmem tb;
  if (MULTI) lj_load_table(tb, tab, ntypes);
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= A.n) return;
  const int nn = min(A.nnb[i], A.maxnb);
  const float4 pi = A.posf[i];
  const int cp = A.cellpack[i];
  const int ti = __float_as_int(pi.w);
  float fx = 0.f, fy = 0.f, fz = 0.f, cfx = 0.f, cfy = 0.f, cfz = 0.f, e = 0.f, ce = 0.f;
  float v[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const ListRows<1, 4> L(A.nbr, i, 0, A.stride, nn);
  const GlobalFetch fetch{A.posf};
  uint32_t ent[4], nxt[4];
  if (L.nrow > 0) L.load(0, ent);
  for (int r = 0; r < L.nrow; ++r) {
    if (r + 1 < L.nrow) L.load(r + 1, nxt);
    float4 pj[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (!L.valid(r, q)) ent[q] = L.standin;
      pj[q] = fetch(ent[q], ent[q] & GBMD_IDX_MASK);
    }
    float rx = 0.f, ry = 0.f, rz = 0.f, re = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t j = ent[q] & GBMD_IDX_MASK;
      const GeomF G = geom_f(ent[q], pj[q], pi, A.g);
      float sig2, eps24, eps4, ecut, rlo, rhi;
      int pid = 0;
      if (MULTI) {
        pid = ti * ntypes + __float_as_int(pj[q].w);
        const float4 a = tb.a[pid];
        const float2 b = tb.b[pid];
        sig2 = a.x; eps24 = a.y; eps4 = a.z; ecut = a.w; rlo = b.x; rhi = b.y;
      } else {
        sig2 = P.sig2; eps24 = P.eps24; eps4 = P.eps4; ecut = P.ecut; rlo = P.rc2lo; rhi = P.rc2hi;
      }
      bool in = G.d2 < rlo;
      if (!in && G.d2 <= rhi && L.valid(r, q))
        in = exact_inside(A.posd, i, j, ent[q] >> GBMD_IDX_BITS, cp, A.g, MULTI ? rcmax2 : P.rc2,
                          MULTI ? tb.r[pid] : 0.0);
      float r2i;
      asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r2i) : "f"(G.d2));
      const float s2 = sig2 * r2i;
      const float s6 = s2 * s2 * s2;
      const float s12 = s6 * s6;
      const float fpair = eps24 * fmaf(2.f, s12, -s6) * r2i;  // -(dE/dr)/r
      if (in) {
        const float gx = fpair * G.dx, gy = fpair * G.dy, gz = fpair * G.dz;
        rx -= gx;
        ry -= gy;
        rz -= gz;
        fix_add(acc + j, fix_q(gx, X.f, FIX_PAIR_LIMIT, X.err));
        fix_add(acc + cap + j, fix_q(gy, X.f, FIX_PAIR_LIMIT, X.err));
        fix_add(acc + 2 * cap + j, fix_q(gz, X.f, FIX_PAIR_LIMIT, X.err));
        if (EV) {
          const float eh = 0.5f * fmaf(eps4, s12 - s6, -ecut);
          const float h = 0.5f * fpair;
          const float w[6] = {h * G.dx * G.dx, h * G.dy * G.dy, h * G.dz * G.dz,
                              h * G.dx * G.dy, h * G.dx * G.dz, h * G.dy * G.dz};
          re += eh;
          fix_add(acc + 3 * cap + j, fix_q(eh, X.e, FIX_PAIR_LIMIT, X.err));
#pragma unroll
          for (int k = 0; k < 6; ++k) {
            v[k] += w[k];
            fix_add(acc + (4 + k) * cap + j, fix_q(w[k], X.v, FIX_PAIR_LIMIT, X.err));
          }
        }
      }
    }
    kahan_add(fx, cfx, rx);
    kahan_add(fy, cfy, ry);
    kahan_add(fz, cfz, rz);
    if (EV) kahan_add(e, ce, re);
#pragma unroll
    for (int q = 0; q < 4; ++q) ent[q] = nxt[q];
  }
  fix_add(acc + i, fix_q(fx - cfx, X.f, FIX_SUM_LIMIT, X.err));
  fix_add(acc + cap + i, fix_q(fy - cfy, X.f, FIX_SUM_LIMIT, X.err));
  fix_add(acc + 2 * cap + i, fix_q(fz - cfz, X.f, FIX_SUM_LIMIT, X.err));
  if (EV) {
    fix_add(acc + 3 * cap + i, fix_q(e - ce, X.e, FIX_SUM_LIMIT, X.err));
#pragma unroll
    for (int k = 0; k < 6; ++k) fix_add(acc + (4 + k) * cap + i, fix_q(v[k], X.v, FIX_SUM_LIMIT, X.err));
  }
}

template <bool EV>
__global__ void __launch_bounds__(256) k_h3_epilogue(PairArgs A, long long* __restrict__ acc, int64_t cap,
                                                     FixScale X, const float* __restrict__ epf) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= A.n) return;
  double f[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    f[d] = (double)acc[d * cap + i] * X.inv_f;
    acc[d * cap + i] = 0;
  }
  const int t = __float_as_int(A.posf[i].w);
  const float im = A.inv_massf[t];
  double o[9];
  double epv = 0.0;
  if (EV) {
    epv = (double)acc[3 * cap + i] * X.inv_e + (epf ? (double)epf[i] : 0.0);
    acc[3 * cap + i] = 0;
    float v[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      v[k] = (float)((double)acc[(4 + k) * cap + i] * X.inv_v);
      acc[(4 + k) * cap + i] = 0;
    }
    vir9(v, o);
  }
  atom_epilogue<true>(A, i, t, 0., 0., 0., (float)f[0] * im, (float)f[1] * im, (float)f[2] * im, epv,
                      EV ? o : nullptr);
}

// Newton-3 eam_alloy (eam_symmetry: eam_force_op_multimat.h L162-169 rho_j
// scatter, L305-338 reaction force): the same per-pair FP32 expressions as
// k_eam_rho_mixed / k_eam_force_mixed on the half list.  The density pass
// adds rho_tj(r) to i's own sum and rho_ti(r) to j's fixed-point plane (the
// energy plane, free until the force pass); k_eam_embed_half turns the sums
// into F'(rho) (and F(rho)); the force pass adds u_ij psi'_ij / r to i and
// its opposite to j, half of phi to both, the pair virial to both.
template <bool SINGLE>
__global__ void __launch_bounds__(256, 4) k_eam_rho_half(PairArgs A, EamDev E, long long* __restrict__ racc,
                                                         FixScale X) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= A.n) return;
  const int nn = min(A.nnb[i], A.maxnb);
  const float4 pi = A.posf[i];
  const int cp = A.cellpack[i];
  const int ti = SINGLE ? 0 : __float_as_int(pi.w);
  const int nr = E.nr, nr1 = E.nr + 1;
  float rho = 0.f, crho = 0.f;
  const ListRows<1, 4> L(A.nbr, i, 0, A.stride, nn);
  const GlobalFetch fetch{A.posf};
  uint32_t ent[4], nxt[4];
  if (L.nrow > 0) L.load(0, ent);
  for (int r = 0; r < L.nrow; ++r) {
    if (r + 1 < L.nrow) L.load(r + 1, nxt);
    float4 pj[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (!L.valid(r, q)) ent[q] = L.standin;
      pj[q] = fetch(ent[q], ent[q] & GBMD_IDX_MASK);
    }
    float rr = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t j = ent[q] & GBMD_IDX_MASK;
      const GeomF G = geom_f(ent[q], pj[q], pi, A.g);
      bool in = G.d2 < E.rc2lo;
      if (!in && G.d2 <= E.rc2hi && L.valid(r, q))
        in = exact_inside(A.posd, i, j, ent[q] >> GBMD_IDX_BITS, cp, A.g, E.rcut2, 0.0);
      const float rd = G.d2 * rsqrtf(G.d2);
      float t;
      const int m = knot_f(rd, E.rdrf, nr, t);
      const int tj = SINGLE ? 0 : __float_as_int(pj[q].w);
      const float vj = spline_val(__ldg(&E.rhor4[tj * nr1 + m]), t);
      const float vi = (SINGLE || ti == tj) ? vj : spline_val(__ldg(&E.rhor4[ti * nr1 + m]), t);
      rr += in ? vj : 0.f;
      if (in) fix_add(racc + j, fix_q(vi, X.r, FIX_PAIR_LIMIT, X.err));
    }
    kahan_add(rho, crho, rr);
#pragma unroll
    for (int q = 0; q < 4; ++q) ent[q] = nxt[q];
  }
  fix_add(racc + i, fix_q(rho - crho, X.r, FIX_SUM_LIMIT, X.err));
}

// Rho2EmbOp / eam_alloy_fEmbed on the summed densities (the embedding of
// eam_rho_atom): F'(rho), F(rho) on energy steps, linear continuation above
// rhomax; the density plane is cleared for the energies of the force pass.
template <bool EV, bool SINGLE>
__global__ void __launch_bounds__(256) k_eam_embed_half(PairArgs A, EamDev E, long long* __restrict__ racc,
                                                        FixScale X, float* __restrict__ fpf, float* __restrict__ epf,
                                                        float4* __restrict__ pfp) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= A.n) return;
  const float R = (float)((double)racc[i] * X.inv_r);
  racc[i] = 0;
  const float4 pi = A.posf[i];
  const int ti = SINGLE ? 0 : __float_as_int(pi.w);
  float q = fmaf(R, E.rdrhof, 1.0f);
  int m = (int)q;
  m = max(1, min(m, E.nrho - 1));
  q = fminf(q - (float)m, 1.0f);
  const float4 c = __ldg(&E.frho4[(SINGLE ? 0 : ti * (E.nrho + 1)) + m]);
  const float fp = spline_der(c, q, E.rdrhof);
  fpf[i] = fp;
  if (SINGLE) pfp[i] = make_float4(pi.x, pi.y, pi.z, fp);
  if (EV) {
    float phi = spline_val(c, q);
    if (R > E.rhomaxf) phi = fmaf(fp, R - E.rhomaxf, phi);
    epf[i] = phi;
  }
}

template <bool EV, bool SINGLE>
__global__ void __launch_bounds__(256, EV ? 1 : 4) k_eam_force_half(PairArgs A, EamDev E,
                                                                    const float* __restrict__ fpf,
                                                                    const float4* __restrict__ pfp,
                                                                    long long* __restrict__ acc, int64_t cap,
                                                                    FixScale X) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= A.n) return;
  const int nn = min(A.nnb[i], A.maxnb);
  const float4 pi = A.posf[i];
  const int cp = A.cellpack[i];
  const float fpi = fpf[i];
  const int ti = SINGLE ? 0 : __float_as_int(pi.w);
  const int nr = E.nr, nr1 = E.nr + 1;
  const float rdr = E.rdrf;
  float fx = 0.f, fy = 0.f, fz = 0.f, cfx = 0.f, cfy = 0.f, cfz = 0.f, e = 0.f, ce = 0.f;
  float v[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const ListRows<1, 4> L(A.nbr, i, 0, A.stride, nn);
  const GlobalFetch fetch{SINGLE ? pfp : A.posf};
  uint32_t ent[4], nxt[4];
  if (L.nrow > 0) L.load(0, ent);
  for (int r = 0; r < L.nrow; ++r) {
    if (r + 1 < L.nrow) L.load(r + 1, nxt);
    float4 pj[4];
    float fpj[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (!L.valid(r, q)) ent[q] = L.standin;
      const uint32_t j = ent[q] & GBMD_IDX_MASK;
      pj[q] = fetch(ent[q], j);
      fpj[q] = SINGLE ? pj[q].w : __ldg(&fpf[j]);
    }
    float rx = 0.f, ry = 0.f, rz = 0.f, re = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t j = ent[q] & GBMD_IDX_MASK;
      const GeomF G = geom_f(ent[q], pj[q], pi, A.g);
      bool in = G.d2 < E.rc2lo;
      if (!in && G.d2 <= E.rc2hi && L.valid(r, q))
        in = exact_inside(A.posd, i, j, ent[q] >> GBMD_IDX_BITS, cp, A.g, E.rcut2, 0.0);
      const float rs = rsqrtf(G.d2);
      const float rd = G.d2 * rs;
      float t;
      const int m = knot_f(rd, rdr, nr, t);
      const int tj = SINGLE ? 0 : __float_as_int(pj[q].w);
      const float4 dj = __ldg(&E.rhod4[tj * nr1 + m]);
      const float4 cz = __ldg(&E.z2r4[z2r_index_d(ti, tj) * nr1 + m]);
      const float rhojp = fmaf(fmaf(dj.x, t, dj.y), t, dj.z);
      float rhoip = rhojp;
      if (!SINGLE && ti != tj) {
        const float4 di = __ldg(&E.rhod4[ti * nr1 + m]);
        rhoip = fmaf(fmaf(di.x, t, di.y), t, di.z);
      }
      const float t1 = fmaf(cz.x, t, cz.y);
      const float z2 = fmaf(fmaf(t1, t, cz.z), t, cz.w);
      const float z2d = fmaf(fmaf(cz.x, t, t1 + t1), t, cz.z);
      const float phi = z2 * rs;
      const float phip = fmaf(z2d * rdr, rs, -phi * rs);
      const float psip = fmaf(fpi, rhojp, fmaf(fpj[q], rhoip, phip));
      const float fpair = in ? psip * rs : 0.f;
      const float gx = G.dx * fpair, gy = G.dy * fpair, gz = G.dz * fpair;
      rx += gx;
      ry += gy;
      rz += gz;
      if (in) {
        fix_add(acc + j, fix_q(-gx, X.f, FIX_PAIR_LIMIT, X.err));
        fix_add(acc + cap + j, fix_q(-gy, X.f, FIX_PAIR_LIMIT, X.err));
        fix_add(acc + 2 * cap + j, fix_q(-gz, X.f, FIX_PAIR_LIMIT, X.err));
        if (EV) {
          const float eh = 0.5f * phi;
          const float h = -0.5f * fpair;
          const float w[6] = {h * G.dx * G.dx, h * G.dy * G.dy, h * G.dz * G.dz,
                              h * G.dx * G.dy, h * G.dx * G.dz, h * G.dy * G.dz};
          re += eh;
          fix_add(acc + 3 * cap + j, fix_q(eh, X.e, FIX_PAIR_LIMIT, X.err));
#pragma unroll
          for (int k = 0; k < 6; ++k) {
            v[k] += w[k];
            fix_add(acc + (4 + k) * cap + j, fix_q(w[k], X.v, FIX_PAIR_LIMIT, X.err));
          }
        }
      }
    }
    kahan_add(fx, cfx, rx);
    kahan_add(fy, cfy, ry);
    kahan_add(fz, cfz, rz);
    if (EV) kahan_add(e, ce, re);
#pragma unroll
    for (int q = 0; q < 4; ++q) ent[q] = nxt[q];
  }
  fix_add(acc + i, fix_q(fx - cfx, X.f, FIX_SUM_LIMIT, X.err));
  fix_add(acc + cap + i, fix_q(fy - cfy, X.f, FIX_SUM_LIMIT, X.err));
  fix_add(acc + 2 * cap + i, fix_q(fz - cfz, X.f, FIX_SUM_LIMIT, X.err));
  if (EV) {
    fix_add(acc + 3 * cap + i, fix_q(e - ce, X.e, FIX_SUM_LIMIT, X.err));
#pragma unroll
    for (int k = 0; k < 6; ++k) fix_add(acc + (4 + k) * cap + i, fix_q(v[k], X.v, FIX_SUM_LIMIT, X.err));
  }
}

// the power of two at or above x (at least 2^-60, which keeps the FP32
// scales finite: all-zero tables give zero contributions at any scale)
static double pow2_at_least(double x) {
  return std::ldexp(1.0, (int)std::ceil(std::log2(std::max(x, 0x1p-60))));
}

// Power-of-two fixed-point scales of the bounds above, from the LJ table.
static FixScale fix_scales(const gbmd_context* c) {
  double fmax = 0.0, emax = 0.0;
  const int nt = c->pot == GBMD_POT_LJ ? 1 : c->lj.ntypes;
  for (int a = 0; a < nt * nt; ++a) {
    const LJPair& q = c->lj.p[a];
    fmax = std::max(fmax, 24.0 * std::fabs(q.eps) / q.sig);
    emax = std::max(emax, 4.0 * std::fabs(q.eps));
  }
  const double vmax = fmax * c->lj.rcut_max;
  const double bf = pow2_at_least(fmax), be = pow2_at_least(emax), bv = pow2_at_least(vmax);
  FixScale X;
  X.f = (float)std::ldexp(1.0 / bf, 38);
  X.e = (float)std::ldexp(1.0 / be, 38);
  X.v = (float)std::ldexp(1.0 / bv, 38);
  X.inv_f = std::ldexp(bf, -38);
  X.inv_e = std::ldexp(be, -38);
  X.inv_v = std::ldexp(bv, -38);
  X.r = 1.f;
  X.inv_r = 1.0;
  X.err = c->d_err + ERRW_FLAGS;
  return X;
}

// eam_alloy: bounds from the host spline copies over the knots from 0.3 rcut
// to rcut (closer pairs are far from any physical state; their
// contributions still fit below 2^16 times the bounds unless they are
// extreme).  Knot m holds the spline on [m dr, (m+1) dr) with value s[6]
// and slope s[5] / dr at its start.  |psi'| <= 2 max|F'| max|rho'| +
// max|phi'|, doubled; energies half phi; virials that force times rcut.
static FixScale eam_fix_scales(gbmd_context* c) {
  if (!c->eam_fix_ok) {
    const EamDev& E = c->eam;
    const double dr = 1.0 / E.rdr, drho = 1.0 / E.rdrho;
    const size_t kr = (size_t)E.nr + 1, kp = (size_t)E.nrho + 1;
    const size_t m0 = std::max<size_t>(1, (size_t)(0.3 * E.rcut / dr));
    const size_t m1 = std::min(kr - 1, (size_t)(E.rcut / dr) + 1);
    double rho = 0.0, rhop = 0.0, phi = 0.0, phip = 0.0, fp = 0.0;
    for (int e = 0; e < E.nel; ++e) {
      for (size_t m = m0; m <= m1; ++m) {
        const double* s = &c->eam_host_rhor[((size_t)e * kr + m) * 8];
        rho = std::max(rho, std::fabs(s[6]));
        rhop = std::max(rhop, std::fabs(s[5]) / dr);
      }
      for (size_t m = 0; m < kp; ++m)
        fp = std::max(fp, std::fabs(c->eam_host_frho[((size_t)e * kp + m) * 8 + 5]) / drho * E.conv_frho);
    }
    for (int p = 0; p < E.npairs; ++p)
      for (size_t m = m0; m <= m1; ++m) {
        const double* s = &c->eam_host_z2r[((size_t)p * kr + m) * 8];
        const double r = (double)m * dr, z2 = s[6] * E.conv_z2r, z2d = s[5] / dr * E.conv_z2r;
        phi = std::max(phi, std::fabs(z2 / r));
        phip = std::max(phip, std::fabs((z2d - z2 / r) / r));
      }
    const double f = 2.0 * (2.0 * fp * rhop + phip);
    c->eam_fix_bound[0] = pow2_at_least(2.0 * rho);
    c->eam_fix_bound[1] = pow2_at_least(f);
    c->eam_fix_bound[2] = pow2_at_least(phi);
    c->eam_fix_bound[3] = pow2_at_least(f * E.rcut);
    c->eam_fix_ok = true;
  }
  const double* b = c->eam_fix_bound;
  FixScale X;
  X.r = (float)std::ldexp(1.0 / b[0], 38);
  X.f = (float)std::ldexp(1.0 / b[1], 38);
  X.e = (float)std::ldexp(1.0 / b[2], 38);
  X.v = (float)std::ldexp(1.0 / b[3], 38);
  X.inv_r = std::ldexp(b[0], -38);
  X.inv_f = std::ldexp(b[1], -38);
  X.inv_e = std::ldexp(b[2], -38);
  X.inv_v = std::ldexp(b[3], -38);
  X.err = c->d_err + ERRW_FLAGS;
  return X;
}

template <bool EV, bool SINGLE>
static void launch_eam_newton3(gbmd_context* c, const PairArgs& A, int part, unsigned grid, int B) {
  cudaStream_t s = c->stream;
  const FixScale X = eam_fix_scales(c);
  long long* racc = c->h3acc + 3 * c->cap;  // the energy plane, free until the force pass
  if (part != 2) {
    k_eam_rho_half<SINGLE><<<grid, B, 0, s>>>(A, c->eam, racc, X);
    k_eam_embed_half<EV, SINGLE><<<grid, B, 0, s>>>(A, c->eam, racc, X, c->fpf, c->epf, c->pfp);
  }
  if (part != 1) {
    k_eam_force_half<EV, SINGLE><<<grid, B, 0, s>>>(A, c->eam, c->fpf, c->pfp, c->h3acc, c->cap, X);
    k_h3_epilogue<EV><<<grid, B, 0, s>>>(A, c->h3acc, c->cap, X, EV ? c->epf : nullptr);
  }
}

template <bool EV>
static int launch_newton3(gbmd_context* c, const PairArgs& A, int part) {
  if (A.n == 0) return GBMD_OK;
  const int B = 256;
  const unsigned grid = (unsigned)((A.n + B - 1) / B);
  if (c->pot == GBMD_POT_EAM_ALLOY) {
    if (c->eam.nel == 1) launch_eam_newton3<EV, true>(c, A, part, grid, B);
    else launch_eam_newton3<EV, false>(c, A, part, grid, B);
    return GBMD_OK;
  }
  if (part == 1) return GBMD_OK;
  cudaStream_t s = c->stream;
  const FixScale X = fix_scales(c);
  if (c->pot == GBMD_POT_LJ) {
    const LJPair& q = c->lj.p[0];
    LJF P{q.sig2f, q.eps24f, q.eps4f, q.ecutf, q.rc2lo, q.rc2hi, q.rc2, q.rc};
    k_lj_half<EV, false><<<grid, B, 0, s>>>(A, P, nullptr, 1, c->lj.rcut_max2, c->h3acc, c->cap, X);
  } else {
    LJF P{};
    k_lj_half<EV, true><<<grid, B, 0, s>>>(A, P, c->lj_tab_d, c->lj.ntypes, c->lj.rcut_max2, c->h3acc, c->cap, X);
  }
  k_h3_epilogue<EV><<<grid, B, 0, s>>>(A, c->h3acc, c->cap, X, nullptr);
  return GBMD_OK;
}

// ---------------------------------------------------------------------------
// dispatch
// ---------------------------------------------------------------------------
template <int T, int V, bool EV, bool PIECE>
static void launch_mixed_TV(gbmd_context* c, const PairArgs& A, int part) {
  const int B = c->block;
  const unsigned grid = (unsigned)(((A.n - A.i0) * T + B - 1) / B);
  const int Bd = c->block_rho ? c->block_rho : B;  // density kernels
  const unsigned gridd = (unsigned)(((A.n - A.i0) * T + Bd - 1) / Bd);
  cudaStream_t s = c->stream;
  if (c->pot == GBMD_POT_LJ) {
    if (part == 1) return;
    const LJPair& q = c->lj.p[0];
    LJF P{q.sig2f, q.eps24f, q.eps4f, q.ecutf, q.rc2lo, q.rc2hi, q.rc2, q.rc};
    k_lj_mixed<T, V, EV, false, PIECE><<<grid, B, 0, s>>>(A, P, nullptr, 1, c->lj.rcut_max2);
  } else if (c->pot == GBMD_POT_LJ_MULTI) {
    if (part == 1) return;
    LJF P{};
    k_lj_mixed<T, V, EV, true, PIECE><<<grid, B, 0, s>>>(A, P, c->lj_tab_d, c->lj.ntypes, c->lj.rcut_max2);
  } else if (c->eam.nel == 1) {
    if (part != 2) k_eam_rho_mixed<T, V, EV, true, PIECE><<<gridd, Bd, 0, s>>>(A, c->eam, c->fpf, c->epf, c->pfp);
    if (part != 1) k_eam_force_mixed<T, V, EV, true, PIECE><<<grid, B, 0, s>>>(A, c->eam, c->fpf, c->epf, c->pfp);
  } else {
    if (part != 2) k_eam_rho_mixed<T, V, EV, false, PIECE><<<gridd, Bd, 0, s>>>(A, c->eam, c->fpf, c->epf, c->pfp);
    if (part != 1) k_eam_force_mixed<T, V, EV, false, PIECE><<<grid, B, 0, s>>>(A, c->eam, c->fpf, c->epf, c->pfp);
  }
}

// Staged launch (one lane per atom, 4 entries per load): blocks of K home
// cells along x; K gives about 0.8 * block atoms per block, and the staged
// capacity is 1.4 times the mean neighbourhood of (K+2) x 3 x 3 cells (a
// denser block falls back to global gathers).
// Raise the dynamic shared-memory limit of the staged kernels once, outside
// any stream capture (the attribute is per kernel, not per launch).
static constexpr int STAGED_MAX_SMEM = 200 * 1024;

int configure_staged_kernels() {
  cudaError_t e = cudaSuccess;
  auto set = [&](const void* f) {
    const cudaError_t r = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, STAGED_MAX_SMEM);
    if (r != cudaSuccess) e = r;
  };
  set((const void*)k_lj_staged<false, false>);
  set((const void*)k_lj_staged<true, false>);
  set((const void*)k_lj_staged<false, true>);
  set((const void*)k_lj_staged<true, true>);
  set((const void*)k_eam_rho_staged<false>);
  set((const void*)k_eam_rho_staged<true>);
  set((const void*)k_eam_force_staged<false>);
  set((const void*)k_eam_force_staged<true>);
  set((const void*)k_eam_rho_bonds_staged);
  set((const void*)k_eam_force_bonds_staged);
  return e == cudaSuccess ? GBMD_OK : GBMD_ERR_CUDA;
}

template <bool EV>
static bool launch_staged(gbmd_context* c, const PairArgs& A, int part) {
  const bool lj = c->pot == GBMD_POT_LJ || c->pot == GBMD_POT_LJ_MULTI;
  if (!lj && !(c->pot == GBMD_POT_EAM_ALLOY && c->eam.nel == 1)) return false;
  const Grid& g = c->grid;
  const double per_cell = (double)A.n / (double)g.ncells;
  const int B = c->block;
  int K = (int)(0.8 * B / (per_cell > 0.5 ? per_cell : 0.5));
  K = K < 1 ? 1 : (K > g.nc[0] ? g.nc[0] : K);
  int cap = (int)(1.4 * per_cell * 9 * (K + 2)) + 64;
  const int max_cap = STAGED_MAX_SMEM / (int)sizeof(float4);
  if (cap > max_cap) cap = max_cap;
  const size_t smem = (size_t)cap * sizeof(float4);
  const dim3 grid((unsigned)((g.nc[0] + K - 1) / K), (unsigned)g.nc[1], (unsigned)g.nc[2]);
  cudaStream_t s = c->stream;
  if (c->pot == GBMD_POT_LJ) {
    if (part == 1) return true;
    const LJPair& q = c->lj.p[0];
    LJF P{q.sig2f, q.eps24f, q.eps4f, q.ecutf, q.rc2lo, q.rc2hi, q.rc2, q.rc};
    k_lj_staged<EV, false><<<grid, B, smem, s>>>(A, P, nullptr, 1, c->lj.rcut_max2, c->cell_start, K, cap);
  } else if (c->pot == GBMD_POT_LJ_MULTI) {
    if (part == 1) return true;
    LJF P{};
    k_lj_staged<EV, true><<<grid, B, smem, s>>>(A, P, c->lj_tab_d, c->lj.ntypes, c->lj.rcut_max2, c->cell_start,
                                                 K, cap);
  } else if (!EV && c->rho_bonds) {
    if (part != 2)
      k_eam_rho_bonds_staged<<<grid, B, smem, s>>>(A, c->eam, c->fpf, c->pfp, c->cell_start, K, cap);
    if (part != 1) k_eam_force_bonds_staged<<<grid, B, smem, s>>>(A, c->fpf, c->pfp, c->cell_start, K, cap);
  } else {
    if (part != 2)
      k_eam_rho_staged<EV><<<grid, B, smem, s>>>(A, c->eam, c->fpf, c->epf, c->pfp, c->cell_start, K, cap);
    if (part != 1)
      k_eam_force_staged<EV><<<grid, B, smem, s>>>(A, c->eam, c->fpf, c->epf, c->pfp, c->cell_start, K, cap);
  }
  return true;
}

template <int T, bool PIECE>
static void launch_bonds_T(gbmd_context* c, const PairArgs& A, int part) {
  const int64_t threads = (A.n - A.i0) * T;
  const int B = c->block, Bd = std::min(128, c->block_rho ? c->block_rho : B);
  cudaStream_t s = c->stream;
  if (part != 2) k_eam_rho_bonds<T, PIECE><<<(unsigned)((threads + Bd - 1) / Bd), Bd, 0, s>>>(A, c->eam, c->fpf, c->pfp);
  if (part != 1) k_eam_force_bonds<T, PIECE><<<(unsigned)((threads + B - 1) / B), B, 0, s>>>(A, c->fpf, c->pfp);
}

template <bool PIECE>
static void launch_bonds(gbmd_context* c, const PairArgs& A, int part) {
  switch (c->tpa) {
    case 1: launch_bonds_T<1, PIECE>(c, A, part); break;
    case 2: launch_bonds_T<2, PIECE>(c, A, part); break;
    case 4: launch_bonds_T<4, PIECE>(c, A, part); break;
    case 8: launch_bonds_T<8, PIECE>(c, A, part); break;
    default: launch_bonds_T<16, PIECE>(c, A, part); break;
  }
}

// One-element eam_alloy without energies goes through the bond passes; a force
// pass on its own, the way of its density pass (of the whole system, or all
// its pieces).
static bool take_bonds(gbmd_context* c, const PairArgs& A, int part, bool ev) {
  if (c->pot != GBMD_POT_EAM_ALLOY || c->eam.nel != 1) return false;
  const bool can = !ev && !c->newton3 && c->vec == 4 && c->f0 && c->bpair_cap >= (int64_t)(c->maxnb / A.W) * A.stride;
  if (part != 2) c->rho_bonds = can;
  return can && c->rho_bonds;
}

template <bool EV, bool PIECE>
static int launch_mixed_shape(gbmd_context* c, const PairArgs& A, int part) {
  const int key = c->tpa * 8 + c->vec;
  switch (key) {
    case 1 * 8 + 1: launch_mixed_TV<1, 1, EV, PIECE>(c, A, part); break;
    case 1 * 8 + 4: launch_mixed_TV<1, 4, EV, PIECE>(c, A, part); break;
    case 2 * 8 + 1: launch_mixed_TV<2, 1, EV, PIECE>(c, A, part); break;
    case 2 * 8 + 4: launch_mixed_TV<2, 4, EV, PIECE>(c, A, part); break;
    case 4 * 8 + 1: launch_mixed_TV<4, 1, EV, PIECE>(c, A, part); break;
    case 4 * 8 + 4: launch_mixed_TV<4, 4, EV, PIECE>(c, A, part); break;
    case 8 * 8 + 1: launch_mixed_TV<8, 1, EV, PIECE>(c, A, part); break;
    case 8 * 8 + 4: launch_mixed_TV<8, 4, EV, PIECE>(c, A, part); break;
    case 16 * 8 + 4: launch_mixed_TV<16, 4, EV, PIECE>(c, A, part); break;
    case 16 * 8 + 1: launch_mixed_TV<16, 1, EV, PIECE>(c, A, part); break;
    default:
      return set_error(c, GBMD_ERR_INVALID, "unsupported launch: %d lanes x %d entries per atom", c->tpa, c->vec);
  }
  return GBMD_OK;
}

template <bool EV>
static int launch_mixed_E(gbmd_context* c, const PairArgs& A, int part) {
  if (c->newton3) {
    // the half list is laid out as one lane x 4 entries per load
    if (c->tpa != 1 || c->vec != 4)
      return set_error(c, GBMD_ERR_UNSUPPORTED, "Newton-3 half lists need the 1 lane x 4 entries launch");
    return launch_newton3<EV>(c, A, part);
  }
  if (c->staged && c->tpa == 1 && c->vec == 4 && launch_staged<EV>(c, A, part)) return GBMD_OK;
  return launch_mixed_shape<EV, false>(c, A, part);
}

int launch_mixed(gbmd_context* c, const PairArgs& A, int part, bool ev) {
  // a piece of the cell order (the host-step pipeline: no energies, full
  // list, no staging, checked by launch_forces)
  if (A.i0 != 0 || A.n != c->n) {
    if (ev) return set_error(c, GBMD_ERR_INVALID, "atom ranges: no energies or virials");
    if (take_bonds(c, A, part, false)) {
      launch_bonds<true>(c, A, part);
      return GBMD_OK;
    }
    return launch_mixed_shape<false, true>(c, A, part);
  }
  const bool bonds = take_bonds(c, A, part, ev);
  if (bonds && !(c->staged && c->tpa == 1)) {
    launch_bonds<false>(c, A, part);
    return GBMD_OK;
  }
  return ev ? launch_mixed_E<true>(c, A, part) : launch_mixed_E<false>(c, A, part);
}

}  // namespace gbmd
