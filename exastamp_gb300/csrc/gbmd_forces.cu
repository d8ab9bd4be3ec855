// gbmd_forces.cu -- plain-FP64 LJ and eam_alloy pair kernels for sm_103a, and
// the force dispatch (FP64 here, mixed precision in gbmd_mixed.cu).
//
// The functions of the reference, in FP64 throughout:
//   LJ       lennard_jones.h L41-50 + force_op_impl2.hxx L33-68 (e -= ecut, de /= r,
//            fe = de*dr, ep += e/2, vir += -1/2 fe (x) dr)
//   LJ multi pair_potential_force_op_multiparam.h L92-118 (r <= rcut_pair test)
//   EAM      eam_alloy.h L198-313 + eam_force_op_multimat.h L114-343
// dr = (x_j + n*L) - x_i and d2 are rounded exactly like the list builder and the
// oracle, so cutoff membership is identical.  The rest is not the reference's
// arithmetic operation for operation: LJ is a function of 1/d2 where the
// reference divides by r, sums are fused, factors common to all pairs are taken
// at the end, and sqrt and 1/x are gbmd_fp64.cuh's (each within one unit in the
// last place of the correctly rounded value).  A pair's force differs by a few
// units in the last place: against quad precision LJ is off by 1.4e-15 (the
// reference's form: 1.8e-15), Cu by 1.9e-15 (1.9e-15).
//
// The FP64 pipe is the bound: an FP64 instruction of a warp takes 16 cycles
// of an SM, as long as some 60 FP32 or integer ones over its four schedulers.
// So everything that need not be FP64 is not: the cutoff is screened in FP32
// (the mixed kernels' screen, exact outside its band), the knot index and the
// float conversions are integer arithmetic, 1/r comes from an FP32 seed, image
// shifts are added only in border cells, and the virial's six values carry
// their factor at the end.  Cu, 108,000 atoms, with energies and virials:
// density 437 -> 288 us, force 928 -> 577 us; LJ, 256,000
// atoms: 3,456 -> 1,134 us.
#include "gbmd_fp64.cuh"
#include "gbmd_pair_common.cuh"

namespace gbmd {

// Where atom i's pairs start from: its positions and its cell.
struct PairHome {
  double4_32a pd;
  float4 pf;
  int cx, cy, cz, nn;
  bool border;  // some stencil cell lies across the box face
  float slack;
  const uint32_t* row;
  __device__ __forceinline__ PairHome(const PairArgs& A, int64_t i, bool live)
      : pd(make_double4_32a(0., 0., 0., 0.)), pf(make_float4(0.f, 0.f, 0.f, 0.f)), cx(0), cy(0), cz(0), nn(0),
        row(A.nbr + (size_t)i * A.W) {
    if (live) {
      pd = A.posd[i];
      pf = A.posf[i];
      unpack_cell(A.cellpack[i], cx, cy, cz);
      nn = min(A.nnb[i], A.maxnb);
    }
    slack = drift_slack(A, pf);
    border = cx == 0 || cy == 0 || cz == 0 || cx == A.g.nc[0] - 1 || cy == A.g.nc[1] - 1 || cz == A.g.nc[2] - 1;
  }
  // FP64 separation of entry ent and its squared length
  __device__ __forceinline__ double separation(const PairArgs& A, uint32_t ent, double& dx, double& dy,
                                               double& dz) const {
    const double4_32a pj = A.posd[ent & GBMD_IDX_MASK];
    double x = pj.x, y = pj.y, z = pj.z;
    if (border) {
      const uint32_t code = ent >> GBMD_IDX_BITS;
      const int nx = image_of(cx, code_dx(code), A.g.nc[0]), ny = image_of(cy, code_dy(code), A.g.nc[1]),
                nz = image_of(cz, code_dz(code), A.g.nc[2]);
      if (nx) x = __dadd_rn(x, nx > 0 ? A.g.L[0] : -A.g.L[0]);
      if (ny) y = __dadd_rn(y, ny > 0 ? A.g.L[1] : -A.g.L[1]);
      if (nz) z = __dadd_rn(z, nz > 0 ? A.g.L[2] : -A.g.L[2]);
    }
    // the reference's rounding, which the oracle shares
    dx = __dsub_rn(x, pd.x);
    dy = __dsub_rn(y, pd.y);
    dz = __dsub_rn(z, pd.z);
    return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  }
};

// body(entry, type of j): the entries of a group's list within the cutoff,
// every lane its own k = lane, lane + T, ...  A lane runs ahead over the
// entries that the FP32 screen excludes, so a warp takes the FP64 body as
// often as its fullest lane has pairs, not list entries (44 and 54, Cu).
// limits(type): the screen's band and the exact cutoffs of the pair.
struct PairLimits {
  float lo, hi;
  double rc2, rc;  // rc <= 0: no second test
};

template <int T, class Limits, class Body>
__device__ __forceinline__ void for_pairs(const PairArgs& A, const PairHome& H, int64_t i, int lane, Limits limits,
                                          Body body) {
  int k = lane;
  for (;;) {
    uint32_t ent = 0;
    int tj = 0;
    bool found = false;
    while (k < H.nn && !found) {
      ent = __ldg(H.row + list_slot(A, k));
      k += T;
      const float4 pj = A.posf[ent & GBMD_IDX_MASK];
      tj = __float_as_int(pj.w);
      const PairLimits P = limits(tj);
      const float d2 = geom_f(ent, pj, H.pf, A.g).d2;
      found = d2 <= P.hi + H.slack;
      if (found && d2 >= P.lo - H.slack)
        found = exact_inside(A.posd, i, ent & GBMD_IDX_MASK, ent >> GBMD_IDX_BITS, A.cellpack[i], A.g, P.rc2, P.rc);
    }
    if (!found) break;
    body(ent, tj);
  }
}

// Epilogue of a block's atoms i0 .. i0 + blockDim / T: the sums f (3), e and
// the virial xx yy zz xy xz yz (before its factor -1/2) of each group's first
// lane pass to the block's first blockDim / T threads, one atom each, so that
// the FP64 work per atom runs on full warps; the virial rows are written
// contiguously.  A block whose lanes own an atom each keeps f and e in place.
template <int T, bool EV>
__device__ __forceinline__ void block_epilogue_d(const PairArgs& A, int64_t i0, int ti, double f0, double f1,
                                                 double f2, double e, const double* v,
                                                 const double* __restrict__ emb = nullptr) {
  constexpr bool SHARED = T > 1 || EV;
  constexpr int NF = T > 1 ? 4 : 0, NV = NF + (EV ? 6 : 0);
  __shared__ double sums[SHARED ? NV : 1][SHARED ? 256 / T : 1];
  const int nat = (int)blockDim.x / T;
  if constexpr (SHARED) {
    const int a = (int)threadIdx.x / T;
    if (threadIdx.x % T == 0) {
      if constexpr (T > 1) {
        sums[0][a] = f0;
        sums[1][a] = f1;
        sums[2][a] = f2;
        sums[3][a] = e;
      }
      if constexpr (EV) {
#pragma unroll
        for (int q = 0; q < 6; ++q) sums[NF + q][a] = -0.5 * v[q];
      }
    }
    __syncwarp();  // the lanes' lists differ in length
    __syncthreads();
    if constexpr (EV) {
      const int m = A.want_virial ? (int)min((int64_t)nat, A.n - i0) * 9 : 0;
      for (int k = threadIdx.x; k < m; k += blockDim.x)  // row-major 3x3
        A.vir[9 * i0 + k] = sums[NF + (int)((0x254513430ll >> (4 * (k % 9))) & 15)][k / 9];
    }
    if ((int)threadIdx.x >= nat) return;
    if constexpr (T > 1) {
      f0 = sums[0][threadIdx.x];
      f1 = sums[1][threadIdx.x];
      f2 = sums[2][threadIdx.x];
      e = sums[3][threadIdx.x];
    }
  }
  const int64_t i = i0 + threadIdx.x;
  if (i >= A.n) return;
  if (T > 1) ti = __float_as_int(A.posf[i].w);
  if (EV && emb) e += emb[i];
  atom_epilogue<false>(A, i, ti, f0, f1, f2, 0.f, 0.f, 0.f, e, nullptr);
}

// ---------------------------------------------------------------------------
// Lennard-Jones (single parameter set and per-type-pair tables)
// ---------------------------------------------------------------------------
template <int T, bool EV, bool MULTI>
__global__ void __launch_bounds__(256) k_lj(PairArgs A, LJPair P, const LJPair* __restrict__ tab, int ntypes,
                                            double rcmax2) {
  __shared__ double sd[MULTI ? GBMD_MAX_TYPES * GBMD_MAX_TYPES * 4 : 1];
  __shared__ float2 sb[MULTI ? GBMD_MAX_TYPES * GBMD_MAX_TYPES : 1];
  if (MULTI) {
    for (int q = threadIdx.x; q < ntypes * ntypes; q += blockDim.x) {
      const LJPair& p = tab[q];
      sd[4 * q + 0] = p.eps;
      sd[4 * q + 1] = p.sig * p.sig;
      sd[4 * q + 2] = p.rc;
      sd[4 * q + 3] = p.ecut;
      sb[q] = make_float2(p.rc2lo, p.rc2hi);
    }
    __syncthreads();
  }
  const int64_t i0 = A.i0 + blockIdx.x * (int64_t)(blockDim.x / T);
  const int64_t i = i0 + threadIdx.x / T;
  const int lane = (int)threadIdx.x % T;
  const PairHome H(A, i, i < A.n);
  const int ti = __float_as_int(H.pf.w);
  double fx = 0., fy = 0., fz = 0., e = 0.;
  double v[6] = {0., 0., 0., 0., 0., 0.};
  auto limits = [&](int tj) {
    if (!MULTI) return PairLimits{P.rc2lo, P.rc2hi, P.rc2, 0.0};
    const int q = ti * ntypes + tj;
    return PairLimits{sb[q].x, sb[q].y, rcmax2, sd[4 * q + 2]};
  };
  for_pairs<T>(A, H, i, lane, limits, [&](uint32_t ent, int tj) {
    double dx, dy, dz;
    const double d2 = H.separation(A, ent, dx, dy, dz);
    const double* p = sd + (MULTI ? 4 * (ti * ntypes + tj) : 0);
    const double eps = MULTI ? p[0] : P.eps, sig2 = MULTI ? p[1] : P.sig * P.sig;
    const double r2i = inverse(d2);
    const double s2 = sig2 * r2i;
    const double s6 = s2 * s2 * s2;
    const double s12 = s6 * s6;
    const double de = (-24. * eps) * (fma(2., s12, -s6) * r2i);
    fx = fma(de, dx, fx);
    fy = fma(de, dy, fy);
    fz = fma(de, dz, fz);
    if (EV) {
      e += fma(4. * eps, s12 - s6, -(MULTI ? p[3] : P.ecut));
      const double fex = de * dx, fey = de * dy;
      v[0] = fma(fex, dx, v[0]);
      v[1] = fma(fey, dy, v[1]);
      v[2] = fma(de * dz, dz, v[2]);
      v[3] = fma(fex, dy, v[3]);
      v[4] = fma(fex, dz, v[4]);
      v[5] = fma(fey, dz, v[5]);
    }
  });
  fx = group_reduce_d<T>(fx);
  fy = group_reduce_d<T>(fy);
  fz = group_reduce_d<T>(fz);
  if (EV) {
    e = group_reduce_d<T>(e);
#pragma unroll
    for (int q = 0; q < 6; ++q) v[q] = group_reduce_d<T>(v[q]);
  }
  block_epilogue_d<T, EV>(A, i0, ti, fx, fy, fz, 0.5 * e, v);
}

// ---------------------------------------------------------------------------
// eam_alloy: density + embedding (one kernel), force (second kernel)
// ---------------------------------------------------------------------------
template <int T, bool EV>
__global__ void __launch_bounds__(256) k_eam_rho(PairArgs A, EamDev E, double* __restrict__ fpd) {
  const int64_t i0 = A.i0 + blockIdx.x * (int64_t)(blockDim.x / T);
  int64_t i = i0 + threadIdx.x / T;
  double rho = 0.;
  {
    const PairHome H(A, i, i < A.n);
    auto limits = [&](int) { return PairLimits{E.rc2lo, E.rc2hi, E.rcut2, 0.0}; };
    for_pairs<T>(A, H, i, (int)threadIdx.x % T, limits, [&](uint32_t ent, int tj) {
      double dx, dy, dz, y, q;
      const double r = root<false>(H.separation(A, ent, dx, dy, dz), y);
      const int m = r_knot_d(fma(r, E.rdr, 1.0), E.nr, q);
      const double* c = E.rhor + ((size_t)tj * (E.nr + 1) + m) * 8;
      rho += ((c[3] * q + c[4]) * q + c[5]) * q + c[6];
    });
  }
  rho = group_reduce_d<T>(rho);
  if (T > 1) {
    __shared__ double sum[T > 1 ? 256 / T : 1];
    if (threadIdx.x % T == 0) sum[threadIdx.x / T] = rho;
    __syncwarp();
    __syncthreads();
    if (threadIdx.x >= blockDim.x / T) return;
    rho = sum[threadIdx.x];
    i = i0 + threadIdx.x;
  }
  if (i >= A.n) return;
  double q = rho * E.rdrho + 1.0;
  int m = (int)q;
  m = max(1, min(m, E.nrho - 1));
  q -= m;
  q = fmin(q, 1.0);
  const double* c = E.frho + ((size_t)__float_as_int(A.posf[i].w) * (E.nrho + 1) + m) * 8;
  double fp = (c[0] * q + c[1]) * q + c[2];
  double phi = ((c[3] * q + c[4]) * q + c[5]) * q + c[6];
  if (rho > E.rhomax) phi += fp * (rho - E.rhomax);
  phi *= E.conv_frho;
  fp *= E.conv_frho;
  fpd[i] = fp;
  if (EV) A.ep_emb[i] = phi;
}

__device__ __forceinline__ int z2r_index(int a, int b) {
  const int irow = a > b ? a : b, icol = a > b ? b : a;
  return irow * (irow + 1) / 2 + icol;
}

template <int T, bool EV>
__global__ void __launch_bounds__(256) k_eam_force(PairArgs A, EamDev E, const double* __restrict__ fpd) {
  const int64_t i0 = A.i0 + blockIdx.x * (int64_t)(blockDim.x / T);
  const int64_t i = i0 + threadIdx.x / T;
  const PairHome H(A, i, i < A.n);
  const int ti = __float_as_int(H.pf.w);
  const double fpi = i < A.n ? fpd[i] : 0.;
  double fx = 0., fy = 0., fz = 0., e = 0.;
  double v[6] = {0., 0., 0., 0., 0., 0.};
  auto limits = [&](int) { return PairLimits{E.rc2lo, E.rc2hi, E.rcut2, 0.0}; };
  for_pairs<T>(A, H, i, (int)threadIdx.x % T, limits, [&](uint32_t ent, int tj) {
    const double fpj = __ldg(&fpd[ent & GBMD_IDX_MASK]);
    double dx, dy, dz, recip, q;
    const double r = root<true>(H.separation(A, ent, dx, dy, dz), recip);
    const int m = r_knot_d(fma(r, E.rdr, 1.0), E.nr, q);
    const double* cj = E.rhor + ((size_t)tj * (E.nr + 1) + m) * 8;
    const double rhojp = (cj[0] * q + cj[1]) * q + cj[2];
    double rhoip = rhojp;
    if (ti != tj) {
      const double* ci = E.rhor + ((size_t)ti * (E.nr + 1) + m) * 8;
      rhoip = (ci[0] * q + ci[1]) * q + ci[2];
    }
    const double* c = E.z2r + ((size_t)z2r_index(ti, tj) * (E.nr + 1) + m) * 8;
    const double z2p = (c[0] * q + c[1]) * q + c[2];
    const double z2 = ((c[3] * q + c[4]) * q + c[5]) * q + c[6];
    const double phi = z2 * recip;
    const double phip = (z2p - phi) * recip;
    const double psip = fma(phip, E.conv_z2r, fma(fpj, rhoip, fpi * rhojp));
    const double fpair = psip * recip;
    fx = fma(dx, fpair, fx);
    fy = fma(dy, fpair, fy);
    fz = fma(dz, fpair, fz);
    if (EV) {
      e += phi;
      const double fex = dx * fpair, fey = dy * fpair;
      v[0] = fma(fex, dx, v[0]);
      v[1] = fma(fey, dy, v[1]);
      v[2] = fma(dz * fpair, dz, v[2]);
      v[3] = fma(fex, dy, v[3]);
      v[4] = fma(fex, dz, v[4]);
      v[5] = fma(fey, dz, v[5]);
    }
  });
  fx = group_reduce_d<T>(fx);
  fy = group_reduce_d<T>(fy);
  fz = group_reduce_d<T>(fz);
  if (EV) {
    e = group_reduce_d<T>(e);
#pragma unroll
    for (int q = 0; q < 6; ++q) v[q] = group_reduce_d<T>(v[q]);
  }
  // the pair energy goes to the thread that finishes the atom, which adds
  // the embedding energy to it
  e *= 0.5 * E.conv_z2r;
  block_epilogue_d<T, EV>(A, i0, ti, fx, fy, fz, e, v, EV ? A.ep_emb : nullptr);
}

// ---------------------------------------------------------------------------
// host dispatch
// ---------------------------------------------------------------------------
PairArgs make_args(gbmd_context* c, const ForceFlags& f) {
  PairArgs A;
  A.i0 = f.i0;
  A.n = f.i1 >= 0 ? f.i1 : c->n;
  A.W = list_width(c);
  A.wsh = log2_of(A.W);
  A.tsh = log2_of(c->tpa);
  A.stride = c->npad * A.W;
  A.nbr = c->nbr;
  A.nnb = c->nnb;
  A.maxnb = c->maxnb;
  A.posf = c->POSF();
  A.posd = c->POSD();
  A.cellpack = c->cellpack;
  A.g = c->grid;
  A.x = c->X();
  A.y = c->Y();
  A.z = c->Z();
  const int o = c->cur ^ 1;
  A.far = (float)(0x1p19 * c->grid_tol);
  A.reach2 = (float)(2.0 * c->grid_reach);
  A.xo = c->rbuf[o];
  A.yo = c->rbuf[o] + c->cap;
  A.zo = c->rbuf[o] + 2 * c->cap;
  A.posf_o = c->posf[o];
  A.posd_o = c->posd[o];
  A.vx = c->VX(); A.vy = c->VY(); A.vz = c->VZ();
  A.ax = c->AX(); A.ay = c->AY(); A.az = c->AZ();
  A.vxo = f.v_out ? f.v_out : A.vx;
  A.vyo = f.v_out ? f.v_out + c->cap : A.vy;
  A.vzo = f.v_out ? f.v_out + 2 * c->cap : A.vz;
  A.f0 = c->f0;
  A.bpair = c->bpair;
  A.ep = c->ep;
  A.ep_emb = c->epd;
  A.vir = c->vir;
  A.type = c->TYPE();
  for (int t = 0; t < GBMD_MAX_TYPES; ++t) {
    A.mass[t] = t < c->ntypes ? c->mass[t] : 1.0;
    A.inv_massf[t] = (float)(1.0 / A.mass[t]);
  }
  A.fuse = f.fuse;
  const bool test = c->fused_trigger && f.fuse == FUSE_PUSH2_PUSH1;
  A.gate = test ? c->d_err + ERRW_GATE : nullptr;
  A.rref = c->rref;
  A.rcap = c->cap;
  A.thr2 = (0.5 * c->skin) * (0.5 * c->skin);
  A.want_energy = f.energy ? 1 : 0;
  A.want_virial = f.virial ? 1 : 0;
  A.dt = f.sp.dt;
  A.dth = f.sp.dth;
  A.dt2h = f.sp.dt2h;
  A.err = c->d_err;
  return A;
}

// part: 0 = the whole force evaluation, 1 = EAM density+embedding only,
// 2 = the final pair kernel only (used by the per-kernel profiler)
template <int T, bool EV>
static void launch_fp64_T(gbmd_context* c, const PairArgs& A, int part) {
  const int B = c->block;
  const unsigned grid = (unsigned)(((A.n - A.i0) * T + B - 1) / B);
  cudaStream_t s = c->stream;
  if (c->pot != GBMD_POT_EAM_ALLOY && part == 1) return;
  if (c->pot == GBMD_POT_LJ) {
    const LJPair& p = c->lj.p[0];
    k_lj<T, EV, false><<<grid, B, 0, s>>>(A, p, nullptr, 1, c->lj.rcut_max2);
  } else if (c->pot == GBMD_POT_LJ_MULTI) {
    k_lj<T, EV, true><<<grid, B, 0, s>>>(A, LJPair{}, c->lj_tab_d, c->lj.ntypes, c->lj.rcut_max2);
  } else {
    if (part != 2) k_eam_rho<T, EV><<<grid, B, 0, s>>>(A, c->eam, c->fpd);
    if (part != 1) k_eam_force<T, EV><<<grid, B, 0, s>>>(A, c->eam, c->fpd);
  }
}

template <bool EV>
static int launch_fp64(gbmd_context* c, const PairArgs& A, int part) {
  switch (c->tpa) {
    case 1: launch_fp64_T<1, EV>(c, A, part); break;
    case 2: launch_fp64_T<2, EV>(c, A, part); break;
    case 4: launch_fp64_T<4, EV>(c, A, part); break;
    case 8: launch_fp64_T<8, EV>(c, A, part); break;
    case 16: launch_fp64_T<16, EV>(c, A, part); break;
    default: return set_error(c, GBMD_ERR_INVALID, "unsupported lanes per atom %d", c->tpa);
  }
  return GBMD_OK;
}

int launch_forces(gbmd_context* c, const ForceFlags& f) {
  if (c->n == 0) return GBMD_OK;
  // every atom type must index the potential's tables (types < ntypes is
  // checked at upload)
  if (c->pot == GBMD_POT_EAM_ALLOY && c->ntypes > c->eam.nel)
    return set_error(c, GBMD_ERR_INVALID, "%d species but the setfl tables hold %d elements", c->ntypes, c->eam.nel);
  if (c->pot == GBMD_POT_LJ_MULTI && c->ntypes > c->lj.ntypes)
    return set_error(c, GBMD_ERR_INVALID, "%d species but the LJ tables cover %d types", c->ntypes, c->lj.ntypes);
  if (!c->list_valid || !c->nbr) return set_error(c, GBMD_ERR_INVALID, "neighbour list not built");
  const bool piece = f.i0 != 0 || f.i1 >= 0;
  if (piece && (f.i0 < 0 || f.i1 < f.i0 || f.i1 > c->n))
    return set_error(c, GBMD_ERR_INVALID, "atom range [%lld, %lld) outside [0, %lld)", (long long)f.i0,
                     (long long)f.i1, (long long)c->n);
  if (piece && (c->newton3 || c->staged || f.fuse == FUSE_PUSH2_PUSH1))
    return set_error(c, GBMD_ERR_INVALID, "atom ranges: full-list kernels without staging or fused first half");
  const PairArgs A = make_args(c, f);
  const bool ev = f.energy || f.virial;
  const bool mixed = c->precision == GBMD_PRECISION_MIXED;
  if (c->newton3 &&
      !(mixed && (c->pot == GBMD_POT_LJ || c->pot == GBMD_POT_LJ_MULTI || c->pot == GBMD_POT_EAM_ALLOY)))
    return set_error(c, GBMD_ERR_UNSUPPORTED,
                     "Newton-3 half lists: LJ potentials and eam_alloy in mixed precision only");
  if (c->newton3 && !c->h3acc) return set_error(c, GBMD_ERR_INVALID, "Newton-3 accumulators not allocated");
  const int part = f.part;
  int rc;
  if (c->pot == GBMD_POT_EAM_JOHNSON || c->pot == GBMD_POT_EAM_SUTTON_CHEN) rc = launch_johnson(c, A, part, ev, mixed);
  else if (mixed) rc = launch_mixed(c, A, part, ev);
  else rc = ev ? launch_fp64<true>(c, A, part) : launch_fp64<false>(c, A, part);
  if (rc) return rc;
  if (f.fuse == FUSE_PUSH2_PUSH1 && part != 1) c->cur ^= 1;
  return GBMD_OK;
}

}  // namespace gbmd
