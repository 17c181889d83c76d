// LK-ball on B200: water sites, water building and its adjoint, and the
// four-term polar / occluder pair potential (tmol/score/lk_ball/potentials:
// water.hh, lk_ball.hh; acceptor bases tmol/score/hbond/identification.hh:26-168).
// Included by ljlk.cu inside namespace tmol_b200, after ScoreArgs and the
// LJ/LK kernels, whose plan (neighbour detection, count-pair tables, work
// items) the LK-ball kernels share.
//
// A plan resolves, once, every water a PoseStack can carry into a "site":
// the coordinate rows of the atoms that place it (donor: heavy atom and
// hydrogen; acceptor: the acceptor and its two base atoms, which may sit in
// bonded blocks) and its torsion / angle.  Per call, one thread per (atom,
// slot) builds the waters; the scoring kernel walks the plan's work items
// like score_kernel, lists the neighbours' heavy atoms, queues the polar /
// occluder pairs in reach and evaluates them 32 at a time; the adjoint
// accumulates d/dcoords and d/dwaters with atomics, and a second pass moves
// d/dwaters onto the placing atoms.

constexpr int LKB_NW = 4;    // waters per polar atom
constexpr int LKB_NPAR = 9;  // per-atom parameters
constexpr int LKB_PAR_PAD = 12;  // their stride in the kernels' table: three vector loads

enum LkbSiteKind : int { kLkbNone = 0, kLkbDonor = 1, kLkbSp2 = 2, kLkbSp3 = 3, kLkbRing = 4 };

template <typename Real>
struct LkbSite {
  int kind;
  int rowA, rowB, rowB0;  // donor: rowA = heavy atom, rowB = hydrogen
  Real tor, ang;
};

template <typename Real>
struct LkbArgs {
  const LkbSite<Real>* sites;  // [n_atoms * 4]
  int64_t n_sites;
  const int* active;  // the occupied sites (kind != none), ascending
  int64_t n_active;
  const Real* waters;   // [n_atoms][4][3]
  Real* waters_out;
  const Real* dwaters;  // adjoint in
  Real* dwaters_out;    // adjoint out
  const int* npol;      // [nbt]
  const int* nocc;
  const int* hbase;     // [P*B] (rotamer plans: [R]) first heavy record of each block (rotamer)
  const Real* par;      // [nbt][A][12], 9 used
  Real water_dist, hbond_dis, hbond_oh, hbond_h, max_dis;
};

// ---------------------------------------------------------------------------
// plan time: sites

struct LkbTables {
  const int32_t* irc;          // [P][B][C][2]
  const int32_t* all_bonds;    // [nbt][NB][3]
  const int32_t* ranges;       // [nbt][A][2]
  int NB, NT;
  const int32_t* tile_n_donH;  // [nbt][NT]
  const int32_t* tile_n_acc;
  const int32_t* tile_donH;    // [nbt][NT][32]
  const int32_t* tile_donH_hvy;
  const int32_t* tile_which;
  const int32_t* tile_acc;
  const int32_t* tile_hyb;
  const int32_t* tile_nH;
  const int32_t* is_h;         // [nbt][A]
  const int32_t* bt_conn_atom; // [nbt][C]
};

struct LkbAtom {
  int block, bt, atom;
};

__device__ __forceinline__ bool lkb_same(LkbAtom a, LkbAtom b) {
  return a.block == b.block && a.bt == b.bt && a.atom == b.atom;
}

// bonded neighbour k of x (bonded_atom.hh:157-260): intra-block, or the
// partner's connection atom across a connection; atom -1 if unresolved
__device__ inline LkbAtom lkb_bonded(const LkbTables& t, const int* blk_bt, int p, int B, int C, LkbAtom x,
                                     int bidx) {
  const int32_t* e = t.all_bonds + ((int64_t)x.bt * t.NB + bidx) * 3;
  LkbAtom r = {x.block, x.bt, e[1]};
  if (e[1] >= 0) return r;
  if (e[2] < 0 || e[2] >= C) return LkbAtom{-1, -1, -1};
  const int32_t* c = t.irc + (((int64_t)p * B + x.block) * C + e[2]) * 2;
  if (c[1] < 0 || c[1] >= C || c[0] < 0 || c[0] >= B) return LkbAtom{-1, -1, -1};
  r.block = c[0];
  r.bt = blk_bt[p * B + c[0]];
  if (r.bt < 0) return LkbAtom{-1, -1, -1};
  r.atom = t.bt_conn_atom[(int64_t)r.bt * C + c[1]];
  return r;
}

__device__ __forceinline__ bool lkb_is_h(const LkbTables& t, int A, LkbAtom x) {
  return x.atom >= 0 && x.atom < A && t.is_h[(int64_t)x.bt * A + x.atom];
}

// an atom's bond range, clamped to the table
__device__ __forceinline__ void lkb_range(const LkbTables& t, int A, LkbAtom x, int& lo, int& hi) {
  lo = hi = 0;
  if (x.atom < 0 || x.atom >= A) return;
  const int32_t* r = t.ranges + ((int64_t)x.bt * A + x.atom) * 2;
  lo = r[0] < 0 ? 0 : r[0];
  hi = r[1] > t.NB ? t.NB : r[1];
}

// acceptor bases (identification.hh:32-150); false when the water frame
// is undefined
__device__ inline bool lkb_bases(const LkbTables& t, const int* blk_bt, int p, int B, int C, int A, LkbAtom a,
                                 int hyb, LkbAtom& b, LkbAtom& b0) {
  const LkbAtom none = {-1, -1, -1};
  b = none;
  b0 = none;
  if (hyb < 1 || hyb > 3) return false;
  int lo, hi;
  lkb_range(t, A, a, lo, hi);
  for (int i = lo; i < hi; ++i) {
    LkbAtom o = lkb_bonded(t, blk_bt, p, B, C, a, i);
    if (o.atom >= 0 && !lkb_is_h(t, A, o)) {
      b = o;
      break;
    }
  }
  if (hyb == 1) {
    if (b.atom < 0) return false;
    int lo2, hi2;
    lkb_range(t, A, b, lo2, hi2);
    for (int i = lo2; i < hi2; ++i) {
      LkbAtom o = lkb_bonded(t, blk_bt, p, B, C, b, i);
      if (o.atom < 0) continue;
      if (b.block != a.block && o.block == a.block) continue;
      if (!lkb_same(o, a)) {
        b0 = o;
        break;
      }
    }
    if (b0.atom < 0) return false;
  } else if (hyb == 2) {
    for (int i = lo; i < hi; ++i) {
      LkbAtom o = lkb_bonded(t, blk_bt, p, B, C, a, i);
      if (o.atom >= 0 && !lkb_same(o, b) && lkb_is_h(t, A, o)) {
        b0 = o;
        break;
      }
    }
    if (b0.atom < 0)
      for (int i = lo; i < hi; ++i) {
        LkbAtom o = lkb_bonded(t, blk_bt, p, B, C, a, i);
        if (o.atom >= 0 && !lkb_same(o, b)) {
          b0 = o;
          break;
        }
      }
    if (b0.atom < 0) b0 = b;
  } else {
    if (b.atom < 0) return false;
    for (int i = lo; i < hi; ++i) {
      LkbAtom o = lkb_bonded(t, blk_bt, p, B, C, a, i);
      if (o.atom >= 0 && !lkb_same(o, b) && !lkb_is_h(t, A, o)) {
        b0 = o;
        break;
      }
    }
    if (b0.atom < 0) return false;
  }
  return b.atom >= 0 && !lkb_same(b0, b);
}

// The rotamer-set indexing the sites are built from (the op's own
// arguments, read at plan time): waters are built per rotamer, with atoms of
// other blocks taken from those blocks' first rotamers (water.hh:318-327).
struct LkbRots {
  const int32_t* rot_coord_offset;      // [R]
  const int32_t* pose_ind_for_rot;      // [R]
  const int32_t* block_ind_for_rot;     // [R]
  const int32_t* block_type_ind_for_rot;// [R]
  const int32_t* first_rot_for_block;   // [P][B]
  const int32_t* first_rot_block_type;  // [P][B]
  const int32_t* bt_n_atoms;            // [nbt]
  int R, nbt;
  int64_t N;
};

// x's coordinate row for waters of rotamer (p, b, off); -1 if unresolved
__device__ __forceinline__ int64_t lkb_row(const LkbRots& r, int p, int B, int b, int off, LkbAtom x) {
  if (x.block == b) return (int64_t)off + x.atom;
  const int fr = r.first_rot_for_block[p * B + x.block];
  if (fr < 0 || fr >= r.R) return -1;
  return (int64_t)r.rot_coord_offset[fr] + x.atom;
}

// One thread per rotamer: its water sites, the donor and acceptor waters
// the reference builds per rotamer (gen_pose_waters.impl.hh:112-175;
// water.hh:332-445).  In the pose op every block has one rotamer.
template <typename Real>
__global__ void lkb_sites_kernel(LkbRots rs, int P, int B, int C, int A, LkbTables t,
                                 const Real* tors_sp2, int n_sp2, const Real* tors_sp3, int n_sp3,
                                 const Real* tors_ring, int n_ring, Real ang_sp2, Real ang_sp3, Real ang_ring,
                                 LkbSite<Real>* sites, int* status) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rs.R; r += gridDim.x * blockDim.x) {
    const int bt = rs.block_type_ind_for_rot[r];
    if (bt < 0) continue;
    const int p = rs.pose_ind_for_rot[r], b = rs.block_ind_for_rot[r];
    const int off = rs.rot_coord_offset[r];
    if (bt >= rs.nbt || p < 0 || p >= P || b < 0 || b >= B || off < 0) {
      atomicOr(status, kStIndex);
      continue;
    }
    const int n = rs.bt_n_atoms[bt];
    if ((int64_t)off + n > rs.N) {
      atomicOr(status, kStIndex);
      continue;
    }
    for (int tt = 0; tt < t.NT; ++tt) {
      const int64_t tb = (int64_t)bt * t.NT + tt;
      for (int q = 0; q < t.tile_n_donH[tb]; ++q) {
        const int h = tt * TILE + t.tile_donH[tb * TILE + q];
        const int d = t.tile_donH_hvy[tb * TILE + q];
        const int w = t.tile_which[tb * TILE + q];
        if (d < 0 || d >= n || h < 0 || h >= n || w < 0 || w >= LKB_NW) {
          atomicOr(status, kStIndex);
          continue;
        }
        LkbSite<Real> s;
        s.kind = kLkbDonor;
        s.rowA = off + d;
        s.rowB = off + h;
        s.rowB0 = off + d;
        s.tor = s.ang = 0;
        sites[(int64_t)(off + d) * LKB_NW + w] = s;
      }
      for (int q = 0; q < t.tile_n_acc[tb]; ++q) {
        const int a = tt * TILE + t.tile_acc[tb * TILE + q];
        const int hyb = t.tile_hyb[tb * TILE + q];
        const int nh = t.tile_nH[tb * TILE + q];
        if (a < 0 || a >= n || nh < 0) {
          atomicOr(status, kStIndex);
          continue;
        }
        LkbAtom x = {b, bt, a}, bb, b0;
        if (!lkb_bases(t, rs.first_rot_block_type, p, B, C, A, x, hyb, bb, b0)) continue;
        const int64_t rb = lkb_row(rs, p, B, b, off, bb), rb0 = lkb_row(rs, p, B, b, off, b0);
        if (bb.atom >= rs.bt_n_atoms[bb.bt] || b0.atom >= rs.bt_n_atoms[b0.bt] || rb < 0 || rb0 < 0 ||
            rb >= rs.N || rb0 >= rs.N) {
          atomicOr(status, kStIndex);
          continue;
        }
        const Real* tors = hyb == 1 ? tors_sp2 : (hyb == 2 ? tors_sp3 : tors_ring);
        const int nt = hyb == 1 ? n_sp2 : (hyb == 2 ? n_sp3 : n_ring);
        const Real ang = hyb == 1 ? ang_sp2 : (hyb == 2 ? ang_sp3 : ang_ring);
        for (int w = 0; w < nt && w + nh < LKB_NW; ++w) {
          LkbSite<Real> s;
          s.kind = kLkbDonor + hyb;
          s.rowA = off + a;
          s.rowB = (int)rb;
          s.rowB0 = (int)rb0;
          s.tor = tors[w];
          s.ang = ang;
          sites[(int64_t)(off + a) * LKB_NW + w + nh] = s;
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// water building (water.hh:42-44; gen_coord.hh:40-74) and its adjoint

template <typename Real>
struct LkbFrame {
  Real e0[3], e1[3], e2[3], c[3], nd, nu, v[3];
};

template <typename Real>
__device__ __forceinline__ void lkb_cross(const Real* a, const Real* b, Real* o) {
  o[0] = a[1] * b[2] - a[2] * b[1];
  o[1] = a[2] * b[0] - a[0] * b[2];
  o[2] = a[0] * b[1] - a[1] * b[0];
}

template <typename Real>
__device__ __forceinline__ Real lkb_dot(const Real* a, const Real* b) {
  return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

__device__ __forceinline__ float lkb_sqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double lkb_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float lkb_exp(float x) { return expf(x); }
__device__ __forceinline__ double lkb_exp(double x) { return exp(x); }
__device__ __forceinline__ float lkb_log(float x) { return logf(x); }
__device__ __forceinline__ double lkb_log(double x) { return log(x); }
__device__ __forceinline__ void lkb_sincos(float x, float* s, float* c) { sincosf(x, s, c); }
__device__ __forceinline__ void lkb_sincos(double x, double* s, double* c) { sincos(x, s, c); }

template <typename Real>
__device__ inline void lkb_frame(const Real* A, const Real* Bp, const Real* C, Real dist, Real angle, Real tor,
                                 LkbFrame<Real>& f) {
  Real d[3], u[3];
  for (int i = 0; i < 3; ++i) {
    d[i] = A[i] - Bp[i];
    f.c[i] = C[i] - Bp[i];
  }
  f.nd = lkb_sqrt(lkb_dot(d, d));
  for (int i = 0; i < 3; ++i) f.e0[i] = d[i] / f.nd;
  lkb_cross(f.e0, f.c, u);
  f.nu = lkb_sqrt(lkb_dot(u, u));
  if (f.nu == Real(0)) {
    Real alt[3] = {1, 0, 0};
    if (f.e0[0] == Real(1) || f.e0[0] == Real(-1)) {
      alt[0] = 0;
      alt[1] = 1;
    }
    lkb_cross(f.e0, alt, u);
    f.nu = lkb_sqrt(lkb_dot(u, u));
  }
  for (int i = 0; i < 3; ++i) f.e2[i] = u[i] / f.nu;
  lkb_cross(f.e2, f.e0, f.e1);
  Real sa, ca, st, ct;
  lkb_sincos(Real(3.14159265358979323846) - angle, &sa, &ca);
  lkb_sincos(tor, &st, &ct);
  f.v[0] = dist * ca;
  f.v[1] = dist * sa * ct;
  f.v[2] = dist * sa * st;
}

template <typename Real>
__device__ __forceinline__ void lkb_load3(const Real* c, int64_t row, Real* v) {
  v[0] = c[3 * row];
  v[1] = c[3 * row + 1];
  v[2] = c[3 * row + 2];
}

template <typename Real>
__device__ inline void lkb_site_water(const LkbSite<Real>& s, const Real* coords, Real dist, Real* W) {
  Real A[3], Bv[3];
  lkb_load3(coords, s.rowA, A);
  lkb_load3(coords, s.rowB, Bv);
  if (s.kind == kLkbDonor) {
    Real h[3] = {Bv[0] - A[0], Bv[1] - A[1], Bv[2] - A[2]};
    const Real nh = lkb_sqrt(lkb_dot(h, h));
    for (int i = 0; i < 3; ++i) W[i] = A[i] + dist * (h[i] / nh);
    return;
  }
  Real B0v[3];
  lkb_load3(coords, s.rowB0, B0v);
  if (s.kind == kLkbRing)
    for (int i = 0; i < 3; ++i) Bv[i] = (Bv[i] + B0v[i]) / 2;
  LkbFrame<Real> f;
  lkb_frame(A, Bv, B0v, dist, s.ang, s.tor, f);
  for (int i = 0; i < 3; ++i) W[i] = A[i] + f.v[0] * f.e0[i] + f.v[1] * f.e1[i] + f.v[2] * f.e2[i];
}

// The waters of the occupied sites (the empty slots hold NaN, written
// beforehand as a byte fill)
template <typename Real>
__global__ void lkb_waters_kernel(LkbArgs<Real> k, const Real* coords) {
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < k.n_active;
       j += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = k.active[j];
    const LkbSite<Real> s = k.sites[i];
    Real W[3];
    lkb_site_water(s, coords, k.water_dist, W);
    k.waters_out[3 * i] = W[0];
    k.waters_out[3 * i + 1] = W[1];
    k.waters_out[3 * i + 2] = W[2];
  }
}

// dcoords += the adjoint of each occupied site's water
template <typename Real>
__global__ void lkb_waters_backward_kernel(LkbArgs<Real> k, const Real* coords, Real* dcoords) {
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < k.n_active;
       j += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = k.active[j];
    const LkbSite<Real> s = k.sites[i];
    const Real g[3] = {k.dwaters[3 * i], k.dwaters[3 * i + 1], k.dwaters[3 * i + 2]};
    if (g[0] == Real(0) && g[1] == Real(0) && g[2] == Real(0)) continue;
    Real A[3], Bv[3];
    lkb_load3(coords, s.rowA, A);
    lkb_load3(coords, s.rowB, Bv);
    Real gA[3] = {0, 0, 0}, gB[3] = {0, 0, 0}, gC[3] = {0, 0, 0};
    if (s.kind == kLkbDonor) {
      Real h[3] = {Bv[0] - A[0], Bv[1] - A[1], Bv[2] - A[2]};
      const Real nh = lkb_sqrt(lkb_dot(h, h));
      Real n[3] = {h[0] / nh, h[1] / nh, h[2] / nh};
      Real gn[3] = {k.water_dist * g[0], k.water_dist * g[1], k.water_dist * g[2]};
      const Real sd = lkb_dot(n, gn);
      for (int j = 0; j < 3; ++j) {
        const Real gh = (gn[j] - n[j] * sd) / nh;
        gA[j] = g[j] - gh;
        gB[j] = gh;
      }
      for (int j = 0; j < 3; ++j) {
        atomicAdd(&dcoords[3 * (int64_t)s.rowA + j], gA[j]);
        atomicAdd(&dcoords[3 * (int64_t)s.rowB + j], gB[j]);
      }
      continue;
    }
    Real B0v[3], Bm[3];
    lkb_load3(coords, s.rowB0, B0v);
    for (int j = 0; j < 3; ++j) Bm[j] = s.kind == kLkbRing ? (Bv[j] + B0v[j]) / 2 : Bv[j];
    LkbFrame<Real> f;
    lkb_frame(A, Bm, B0v, k.water_dist, s.ang, s.tor, f);
    // reverse mode through W = A + v0 e0 + v1 e1 + v2 e2
    Real ge0[3], ge1[3], ge2[3], tmp[3], gu[3];
    for (int j = 0; j < 3; ++j) {
      gA[j] = g[j];
      ge0[j] = f.v[0] * g[j];
      ge1[j] = f.v[1] * g[j];
      ge2[j] = f.v[2] * g[j];
    }
    lkb_cross(f.e0, ge1, tmp);  // e1 = e2 x e0
    for (int j = 0; j < 3; ++j) ge2[j] += tmp[j];
    lkb_cross(ge1, f.e2, tmp);
    for (int j = 0; j < 3; ++j) ge0[j] += tmp[j];
    Real sd = lkb_dot(f.e2, ge2);  // e2 = u / |u|
    for (int j = 0; j < 3; ++j) gu[j] = (ge2[j] - f.e2[j] * sd) / f.nu;
    lkb_cross(f.c, gu, tmp);  // u = e0 x c
    for (int j = 0; j < 3; ++j) ge0[j] += tmp[j];
    Real gc[3];
    lkb_cross(gu, f.e0, gc);
    sd = lkb_dot(f.e0, ge0);  // e0 = (A - B) / |A - B|
    for (int j = 0; j < 3; ++j) {
      const Real gd = (ge0[j] - f.e0[j] * sd) / f.nd;
      gA[j] += gd;
      gB[j] = -gd - gc[j];
      gC[j] = gc[j];
    }
    for (int j = 0; j < 3; ++j) {
      atomicAdd(&dcoords[3 * (int64_t)s.rowA + j], gA[j]);
      if (s.kind == kLkbRing) {
        atomicAdd(&dcoords[3 * (int64_t)s.rowB + j], gB[j] / 2);
        atomicAdd(&dcoords[3 * (int64_t)s.rowB0 + j], gB[j] / 2);
      } else {
        atomicAdd(&dcoords[3 * (int64_t)s.rowB + j], gB[j]);
      }
      atomicAdd(&dcoords[3 * (int64_t)s.rowB0 + j], gC[j]);
    }
  }
}

// ---------------------------------------------------------------------------
// the pair potential (lk_ball.hh:34-500)

template <typename Real>
struct LkbParams {
  Real lj_radius, lk_dgfree, lk_lambda, lk_volume, is_donor, is_hydroxyl, is_polarh, is_acceptor, is_carbon_lk;
};

template <typename Real>
__device__ __forceinline__ Real lkb_sq(Real v) {
  return v * v;
}

// lk_fraction: value, d/dJ, d/dWI
template <typename Real, bool GRAD>
__device__ inline Real lkb_fraction(const Real* WI, const Real* J, Real lj_radius_j, Real* dJ, Real* dWI) {
  const Real ramp = Real(3.709);
  Real d2_low = lkb_sq(Real(1.4) + lj_radius_j) - ramp;
  if (d2_low < Real(0)) d2_low = 0;
  Real wsum = 0, gJ[3] = {0, 0, 0}, gW[LKB_NW * 3];
#pragma unroll
  for (int i = 0; i < LKB_NW * 3; ++i) gW[i] = 0;
#pragma unroll
  for (int w = 0; w < LKB_NW; ++w) {
    const Real dl[3] = {J[0] - WI[3 * w], J[1] - WI[3 * w + 1], J[2] - WI[3 * w + 2]};
    const Real d2 = lkb_dot(dl, dl) - d2_low;
    if (isnan(d2)) continue;
    const Real e = lkb_exp(-d2);
    wsum += e;
    if (GRAD)
      for (int i = 0; i < 3; ++i) {
        gJ[i] += 2 * e * dl[i];
        gW[3 * w + i] = -2 * e * dl[i];
      }
  }
  const Real x = -lkb_log(wsum);
  Real frac = 0;
  if (x < Real(0))
    frac = 1;
  else if (x < ramp)
    frac = lkb_sq(Real(1) - lkb_sq(x / ramp));
  if (GRAD) {
    Real df = 0;
    if (x > Real(0) && x < ramp) df = -4 * x * (lkb_sq(ramp) - lkb_sq(x)) / lkb_sq(lkb_sq(ramp));
    const Real inv = wsum != Real(0) ? Real(1) / wsum : Real(1);
    for (int i = 0; i < 3; ++i) dJ[i] = gJ[i] * inv * df;
    for (int i = 0; i < LKB_NW * 3; ++i) dWI[i] = gW[i] * inv * df;
  }
  return frac;
}

// lk_bridge_fraction
template <typename Real, bool GRAD>
__device__ inline Real lkb_bridge(const Real* I, const Real* J, const Real* WI, const Real* WJ, Real water_dist,
                                  Real* dI, Real* dJ, Real* dWI, Real* dWJ) {
  const Real gap = Real(0.5), width = Real(2.6), aover = Real(2.8) * Real(2.6);
  Real wsum = 0;
  if (GRAD)
    for (int i = 0; i < LKB_NW * 3; ++i) dWI[i] = dWJ[i] = 0;
#pragma unroll 1
  for (int a = 0; a < LKB_NW; ++a)
#pragma unroll
    for (int c = 0; c < LKB_NW; ++c) {
      const Real dl[3] = {WI[3 * a] - WJ[3 * c], WI[3 * a + 1] - WJ[3 * c + 1], WI[3 * a + 2] - WJ[3 * c + 2]};
      const Real d2 = lkb_dot(dl, dl) - gap;
      if (isnan(d2)) continue;
      const Real e = lkb_exp(-d2);
      if (GRAD)
        for (int i = 0; i < 3; ++i) {
          dWI[3 * a + i] += 2 * e * dl[i];
          dWJ[3 * c + i] -= 2 * e * dl[i];
        }
      wsum += e;
    }
  const Real x = -lkb_log(wsum);
  Real ofrac, dof = 0;
  if (x > width) {
    ofrac = 0;
  } else if (x > Real(0)) {
    ofrac = lkb_sq(Real(1) - lkb_sq(x / width));
    dof = -4 * x * (lkb_sq(width) - lkb_sq(x)) / lkb_sq(lkb_sq(width));
  } else {
    ofrac = 1;
  }
  const Real dIJ[3] = {I[0] - J[0], I[1] - J[1], I[2] - J[2]};
  const Real base = lkb_dot(dIJ, dIJ) - Real(8.0 / 3.0) * lkb_sq(water_dist);
  const Real ab = base < Real(0) ? -base : base;
  Real afrac, daf = 0;
  if (ab > aover) {
    afrac = 0;
  } else if (ab > Real(0)) {
    afrac = lkb_sq(Real(1) - lkb_sq(base / aover));
    daf = -4 * base * (lkb_sq(aover) - lkb_sq(base)) / lkb_sq(lkb_sq(aover));
  } else {
    afrac = 1;
  }
  if (GRAD) {
    const Real inv = wsum != Real(0) ? Real(1) / wsum : Real(1);
    for (int i = 0; i < 3; ++i) {
      dI[i] = ofrac * daf * 2 * dIJ[i];
      dJ[i] = -ofrac * daf * 2 * dIJ[i];
    }
    for (int i = 0; i < LKB_NW * 3; ++i) {
      dWI[i] *= afrac * dof * inv;
      dWJ[i] *= afrac * dof * inv;
    }
  }
  return ofrac * afrac;
}

template <typename Real, typename K>
__device__ __forceinline__ Real lkb_sigma(const LkbParams<Real>& i, const LkbParams<Real>& j, const K& k) {
  const bool di = i.is_donor != 0, dj = j.is_donor != 0, ai = i.is_acceptor != 0, aj = j.is_acceptor != 0;
  if ((di && aj) || (dj && ai)) {
    if ((di && i.is_hydroxyl != 0) || (dj && j.is_hydroxyl != 0)) return k.hbond_oh;
    return k.hbond_dis;
  }
  if ((i.is_polarh != 0 && aj) || (j.is_polarh != 0 && ai)) return k.hbond_h;
  return i.lj_radius + j.lj_radius;
}

// one direction of lk_isotropic (lk_isotropic.hh:97-236)
template <typename Real>
__device__ inline void lkb_lk_pair(Real dist, int sep, Real sigma, Real ri, Real dgi, Real lami, Real volj,
                                   Real max_dis, bool cc, Real& V, Real& dV) {
  Real d_min = sigma * Real(.89);
  if (cc) d_min = d_min > Real(4.2) ? d_min : Real(4.2);
  const Real n = floor(Real(20) * d_min * d_min);
  const Real close_dmin = lkb_sqrt((n - 29 > Real(0) ? n - 29 : Real(0)) / 20);
  const Real close_dmax = lkb_sqrt((n + 21 < Real(405) ? n + 21 : Real(405)) / 20);
  const Real far_dmax = max_dis, far_dmin = max_dis - Real(1.5);
  const Real weight = sep > 4 ? Real(1) : (sep == 4 ? Real(0.2) : Real(0));
  const Real pref = -volj * dgi / (2 * Real(5.56832799683f) * lami);  // pi^1.5 as a float literal, as tmol has it
  auto f = [&](Real d, Real& v, Real& dv) {
    const Real z = (d - ri) / lami;
    const Real ex = lkb_exp(-z * z);
    v = pref / (d * d) * ex;
    dv = pref * ex * (Real(-2) / (d * d * d) + Real(1) / (d * d) * -(2 * d - 2 * ri) / (lami * lami));
  };
  Real lk = 0, dlk = 0;
  if (dist < close_dmin) {
    Real v, dv;
    f(d_min, v, dv);
    lk = v;
  } else if (dist < close_dmax) {
    Real v0, dv0, v1, dv1;
    f(d_min, v0, dv0);
    f(close_dmax, v1, dv1);
    hermite_V_dV(dist, close_dmin, v0, Real(0), close_dmax, v1, dv1, lk, dlk);
  } else if (dist < far_dmin) {
    f(dist, lk, dlk);
  } else if (dist < far_dmax) {
    Real v0, dv0;
    f(far_dmin, v0, dv0);
    hermite_V_dV(dist, far_dmin, v0, dv0, far_dmax, Real(0), Real(0), lk, dlk);
  }
  V = weight * lk;
  dV = weight * dlk;
}

// lk_ball_score (lk_ball.hh:335-500) for polar I against occluder J: E[4]
// and, with GRAD, the adjoint of g . E onto I, J, WI, WJ (added).  Returns
// 0 when the pair is out of reach (bond separation, distance, no water),
// 1 when evaluated, 2 when evaluated with the water-bridge term.
template <typename Real, bool GRAD, typename K>
__device__ inline int lkb_pair(const Real* I, const Real* J, const Real* WI, const Real* WJ, int sep,
                                const LkbParams<Real>& pi, const LkbParams<Real>& pj, const K& k,
                                Real* E, const Real* g, Real* gI, Real* gJ, Real* gWI, Real* gWJ) {
  E[0] = E[1] = E[2] = E[3] = 0;
  if (sep <= 3) return 0;
  const Real dv[3] = {I[0] - J[0], I[1] - J[1], I[2] - J[2]};
  const Real dist = lkb_sqrt(lkb_dot(dv, dv));
  if (dist >= k.max_dis) return 0;
  if (isnan(WI[0])) return 0;
  const Real sigma = lkb_sigma(pi, pj, k);
  Real iso, diso;
  lkb_lk_pair(dist, sep, sigma, pi.lj_radius, pi.lk_dgfree, pi.lk_lambda, pj.lk_volume, k.max_dis,
              pi.is_carbon_lk != 0 && pj.is_carbon_lk != 0, iso, diso);
  Real fdJ[3], fdWI[LKB_NW * 3];
  const Real fdes = lkb_fraction<Real, GRAD>(WI, J, pj.lj_radius, fdJ, fdWI);
  Real bdI[3] = {0, 0, 0}, bdJ[3] = {0, 0, 0}, bdWI[LKB_NW * 3], bdWJ[LKB_NW * 3];
  Real fov = 0;
  const bool bridged = pj.is_donor != 0 || pj.is_acceptor != 0;
  if (bridged) {
    fov = lkb_bridge<Real, GRAD>(I, J, WI, WJ, k.water_dist, bdI, bdJ, bdWI, bdWJ);
  } else if (GRAD) {
    for (int i = 0; i < LKB_NW * 3; ++i) bdWI[i] = bdWJ[i] = 0;
  }
  E[0] = iso;
  E[1] = iso * fdes;
  E[2] = iso * fov;
  E[3] = fov / 2;
  if (!GRAD) return bridged ? 2 : 1;
  Real u[3] = {0, 0, 0};
  if (dist != Real(0))
    for (int i = 0; i < 3; ++i) u[i] = dv[i] / dist;
  const Real giso = g[0] + g[1] * fdes + g[2] * fov;
  for (int i = 0; i < 3; ++i) {
    gI[i] += giso * diso * u[i] + g[2] * iso * bdI[i] + g[3] * bdI[i] / 2;
    gJ[i] += -giso * diso * u[i] + g[1] * iso * fdJ[i] + g[2] * iso * bdJ[i] + g[3] * bdJ[i] / 2;
  }
  for (int i = 0; i < LKB_NW * 3; ++i) {
    gWI[i] += g[1] * iso * fdWI[i] + g[2] * iso * bdWI[i] + g[3] * bdWI[i] / 2;
    gWJ[i] += g[2] * iso * bdWJ[i] + g[3] * bdWJ[i] / 2;
  }
  return bridged ? 2 : 1;
}

// ---------------------------------------------------------------------------
// scoring kernel: the plan's work items (pose, b1, candidate blocks), the
// neighbour rule as score_kernel applies it, then every polar / occluder
// pair of each neighbouring block pair (intra-block: ordered pairs of
// distinct atoms; inter-block: polars of either block against occluders of
// the other), found by lkb_walk.

template <typename Real>
__device__ __forceinline__ LkbParams<Real> lkb_params(const Real* par, int row) {
  const Quad<Real>* q = reinterpret_cast<const Quad<Real>*>(par) + 3 * (int64_t)row;
  const Quad<Real> u = q[0], v = q[1];
  LkbParams<Real> r;
  r.lj_radius = u.a;
  r.lk_dgfree = u.b;
  r.lk_lambda = u.c;
  r.lk_volume = u.d;
  r.is_donor = v.a;
  r.is_hydroxyl = v.b;
  r.is_polarh = v.c;
  r.is_acceptor = v.d;
  r.is_carbon_lk = q[2].a;
  return r;
}

// An atom's four waters: twelve values, 16-byte aligned where the whole array
// is (`vec`; torch's allocations are).
template <typename Real>
__device__ __forceinline__ void lkb_load_waters(const Real* waters, int64_t row, bool vec, Real* W) {
  const Real* p = waters + row * (LKB_NW * 3);
  if (vec) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const Quad<Real> q = reinterpret_cast<const Quad<Real>*>(p)[k];
      W[4 * k] = q.a;
      W[4 * k + 1] = q.b;
      W[4 * k + 2] = q.c;
      W[4 * k + 3] = q.d;
    }
  } else {
#pragma unroll
    for (int k = 0; k < LKB_NW * 3; ++k) W[k] = p[k];
  }
}

// Adds the gradient on an atom's waters, four values a reduction.
__device__ __forceinline__ void lkb_add_waters(float* dwaters, int64_t row, bool vec, const float* g) {
  float* p = dwaters + row * (LKB_NW * 3);
  if (vec) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float a = g[4 * k], b = g[4 * k + 1], c = g[4 * k + 2], d = g[4 * k + 3];
      if (a != 0.0f || b != 0.0f || c != 0.0f || d != 0.0f)
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p + 4 * k), "f"(a), "f"(b), "f"(c), "f"(d)
                     : "memory");
    }
  } else {
#pragma unroll
    for (int k = 0; k < LKB_NW * 3; ++k)
      if (g[k] != 0.0f) atomicAdd(p + k, g[k]);
  }
}
__device__ __forceinline__ void lkb_add_waters(double* dwaters, int64_t row, bool, const double* g) {
  double* p = dwaters + row * (LKB_NW * 3);
#pragma unroll
  for (int k = 0; k < LKB_NW * 3; ++k)
    if (g[k] != 0.0) atomicAdd(p + k, g[k]);
}

// Pairs in reach wait in two per-warp queues, those whose occluder bridges
// (donor or acceptor: the 4 x 4 water-pair term) and the rest, and are
// evaluated 32 at a time with every lane busy on the same branch.
constexpr int LKB_Q = 64;
// warps per CTA of the LK-ball kernels (launches clamp to it)
constexpr int LKB_MAX_WARPS = 8;

template <bool TAGGED>
struct LkbQueue {
  int rp[LKB_Q], ro[LKB_Q], pi[LKB_Q], oi[LKB_Q];  // coordinate rows; (bt * A + atom) of the polar / occluder
  int tag[TAGGED ? LKB_Q : 1];  // the output row each pair belongs to (tagged queues only)
  uint8_t sep[LKB_Q];
};

// What evaluating a queued pair needs (a compact by-value context).
template <typename Real>
struct LkbEval {
  const Real* coords;
  const Real* waters;
  const Real* par;
  Real* dcoords;  // [n_atoms][3]
  Real* dwaters;  // [n_atoms][4][3]
  bool vec_w, vec_dw;  // 16-byte aligned
  Real water_dist, hbond_dis, hbond_oh, hbond_h, max_dis;
};

template <typename Real>
struct Lkb4 {
  Real v[4];
};

// Evaluates entry `lane` of q when lane < n: returns its four energies and,
// with GRAD, adds the adjoint of w . E to dcoords / dwaters.
// inlined: an out-of-line copy (smaller code) measured 34% slower, its
// calling convention spilling the kernel's state
#ifndef TMOL_B200_LKB_DRAIN_ATTR
#define TMOL_B200_LKB_DRAIN_ATTR __forceinline__
#endif
// two 256-thread CTAs per SM (128 registers): measured faster than one
// (182 registers) and than three (80 registers, spilling)
#ifndef TMOL_B200_LKB_MIN_CTAS
#define TMOL_B200_LKB_MIN_CTAS 2
#endif
// The float64 adjoint does not fit in the 128 registers that two CTAs per SM
// leave a thread (it spilled a kilobyte): one, 16 x 150 residues, gradient 355
// us with two, 251 with one.  Float keeps two (one: 30% slower).
template <typename Real, bool GRAD>
constexpr int lkb_min_ctas = sizeof(Real) == 8 && GRAD ? 1 : TMOL_B200_LKB_MIN_CTAS;

template <typename Real, bool GRAD, typename Queue>
__device__ TMOL_B200_LKB_DRAIN_ATTR Lkb4<Real> lkb_drain(const LkbEval<Real> ev, const Queue& q, int n, int lane,
                                             const Lkb4<Real> w) {
  Lkb4<Real> out = {{0, 0, 0, 0}};
  if (lane >= n) return out;
  const int64_t rp = q.rp[lane], ro = q.ro[lane];
  const int pidx = q.pi[lane], oidx = q.oi[lane], sep = q.sep[lane];
  Real WI[LKB_NW * 3], WJ[LKB_NW * 3];
  Real I[3], J[3];
  lkb_load3(ev.coords, rp, I);
  lkb_load3(ev.coords, ro, J);
  lkb_load_waters(ev.waters, rp, ev.vec_w, WI);
  lkb_load_waters(ev.waters, ro, ev.vec_w, WJ);
  const LkbParams<Real> pp = lkb_params(ev.par, pidx);  // row bt * A + atom
  const LkbParams<Real> po = lkb_params(ev.par, oidx);
  Real gI[3] = {0, 0, 0}, gJ[3] = {0, 0, 0}, gWI[LKB_NW * 3], gWJ[LKB_NW * 3];
  if (GRAD)
#pragma unroll
    for (int c = 0; c < LKB_NW * 3; ++c) gWI[c] = gWJ[c] = 0;
  lkb_pair<Real, GRAD>(I, J, WI, WJ, sep, pp, po, ev, out.v, w.v, gI, gJ, gWI, gWJ);
  if (GRAD) {
    // straight into the caller's gradient: with sums in LJ/LK's padded form and
    // its vector reductions the kernel took 164 us for 64 x 150 residues (161
    // without, before the loops in front were folded), and another pass copied
    // them out
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      if (gI[c] != Real(0)) atomicAdd(&ev.dcoords[3 * rp + c], gI[c]);
      if (gJ[c] != Real(0)) atomicAdd(&ev.dcoords[3 * ro + c], gJ[c]);
    }
    lkb_add_waters(ev.dwaters, rp, ev.vec_dw, gWI);
    lkb_add_waters(ev.dwaters, ro, ev.vec_dw, gWJ);
  }
  return out;
}

// Per-warp queue state: the two queues (plain, bridged) in shared memory,
// their fill (warp-uniform) and the work counters.
template <typename Real, bool TAGGED>
struct LkbWarp {
  LkbQueue<TAGGED>* qs;
  int nq[2];
  int lane;
  unsigned lt_mask;
  unsigned long long n_bp, n_pairs, n_bridge, n_eval;
};

// Where tagged entries' energies go and their weights come from:
// out[t * n + tag] (rotamer op: energies [4, n_pairs], dTdV [4, n_pairs]).
template <typename Real>
struct LkbTagged {
  Real* energies;
  const Real* dTdV;
  int64_t n;
};

// Evaluates full queues (or, with `all`, everything queued) under the
// weights w, adding energies to e4, and shifts what is left to the front.
// TAGGED: each entry's weights and energies are those of its tag's row.
template <typename Real, bool GRAD, bool TAGGED>
__device__ __forceinline__ void lkb_pump(const LkbEval<Real>& ev, LkbWarp<Real, TAGGED>& q, bool all, const Lkb4<Real> w,
                                         Real* e4, const LkbTagged<Real> tg) {
  for (;;) {
    int which, n;
    if (q.nq[0] >= 32) {
      which = 0, n = 32;
    } else if (q.nq[1] >= 32) {
      which = 1, n = 32;
    } else if (all && q.nq[0] > 0) {
      which = 0, n = q.nq[0];
    } else if (all && q.nq[1] > 0) {
      which = 1, n = q.nq[1];
    } else {
      break;
    }
    LkbQueue<TAGGED>& Q = q.qs[which];
    const int lane = q.lane;
    __syncwarp();
    Lkb4<Real> wl = w;
    const int tag = TAGGED && lane < n ? Q.tag[lane] : 0;
    if (TAGGED && GRAD && lane < n)
      for (int c = 0; c < 4; ++c) wl.v[c] = tg.dTdV[(int64_t)c * tg.n + tag];
    const Lkb4<Real> got = lkb_drain<Real, GRAD>(ev, Q, n, lane, wl);
    if (TAGGED) {
      if (!GRAD && lane < n)
        for (int c = 0; c < 4; ++c)
          if (got.v[c] != Real(0)) atomicAdd(&tg.energies[(int64_t)c * tg.n + tag], got.v[c]);
    } else {
      for (int c = 0; c < 4; ++c) e4[c] += got.v[c];
    }
    const int rest = (which ? q.nq[1] : q.nq[0]) - n;
    int a = 0, b = 0, c = 0, d = 0, e = 0, f = 0;
    if (lane < rest) {
      a = Q.rp[n + lane], b = Q.ro[n + lane], c = Q.pi[n + lane], d = Q.oi[n + lane], e = Q.sep[n + lane];
      if (TAGGED) f = Q.tag[n + lane];
    }
    __syncwarp();
    if (lane < rest) {
      Q.rp[lane] = a, Q.ro[lane] = b, Q.pi[lane] = c, Q.oi[lane] = d, Q.sep[lane] = (uint8_t)e;
      if (TAGGED) Q.tag[lane] = f;
    }
    __syncwarp();
    if (which)
      q.nq[1] = rest;
    else
      q.nq[0] = rest;
  }
}

// The rows of a walk: a block (or rotamer), its heavy records and atoms.
struct LkbRows {
  int bt, off, hb, nocc, npol, n_atoms;
};

// One neighbour (a block or rotamer) as a lane sees it.
struct LkbHit {
  bool hit;
  int entry;        // its count-pair table entry; -1: the rows themselves; -2: bond separations do not matter
  int bt, off, hb;  // block type, first coordinate row, first heavy record
  int tag;          // output row (tagged queues)
};

// Heavy atoms of a list of neighbours, a few dozen at a time, and where the
// current 32 neighbours' atoms come from.
constexpr int LKB_LIST = 64;
template <typename Real, bool TAGGED>
struct LkbList {
  Real x[LKB_LIST], y[LKB_LIST], z[LKB_LIST];
  int tf[LKB_LIST];  // atom | kHeavyPolar | kHeavyBridges
  int row[LKB_LIST], par[LKB_LIST], entry[LKB_LIST];
  int tag[TAGGED ? LKB_LIST : 1];
  int hoff[32], off[32], bt[32], ent[32], htag[TAGGED ? 32 : 1];
};
// a float64 kernel with tags fills a CTA's static shared memory to the byte:
// what is added to either struct has to come out of LKB_Q, LKB_LIST or the warps
static_assert(LKB_MAX_WARPS * (2 * sizeof(LkbQueue<true>) + sizeof(LkbList<double, true>)) <= 48 * 1024,
              "static shared memory");

// Whether a squared distance is one below `max`, as the square root decides it
// (in float64 asked only where it could decide otherwise).
__device__ __forceinline__ bool lkb_within(float d2, float max) { return lkb_sqrt(d2) < max; }
__device__ __forceinline__ bool lkb_within(double d2, double max) {
  const double m2 = max * max;
  return d2 < m2 * (1 - 1e-12) || (d2 < m2 * (1 + 1e-12) && lkb_sqrt(d2) < max);
}

// Queues every polar / occluder pair between the rows and the n_cand
// neighbours that `next(first)` yields 32 at a time (each lane one), and
// evaluates full queues under w into e4.  The neighbours' heavy atoms are one
// flat list: each is loaded once with its flags (polar with waters, bridges)
// and culled against the rows' sphere (centre c, reach2 the squared reach),
// and 32 of them at a time, one a lane, meet the rows: a lane first finds its
// pairs as bits (in reach, not excluded, weight 0.2), in loops whose loads do
// not wait for one another, then the warp queues a pair of each lane at a time
// until none has one left.  Pairs of the rows' own block and of count-pair
// partners have their exclusions from the plan's masks, a rotamer's partners
// (PMASK false) their bond separations.
// What bounds it: latency and issue of the evaluation, and beside the adjoint
// the instruction cache: the rows' loops are unrolled for the energies alone
// (64 x 150 residues, energies + gradients: 157 us with them unrolled by four,
// 152 by two, 148 not at all).  Times of the scoring kernel where pairs were
// enumerated one by one, with index arithmetic and eight loads each; where every
// row was voted on and queued in both directions in turn, its record and masks
// loaded in between; and now: 64 x 150 residues, energies + gradients 196, 164
// and 148 us; rotamers of 4 x 100 residues, ten a block, energies 151, 169 and
// 106 us; one pose of 100 residues, energies 37, 35 and 26 us; 4 x 100 in
// float64, energies 101, 128 and 102 us; one residue 7.5, 14.7 and 7.8-8.8 us.
template <typename Real, bool GRAD, bool TAGGED, bool COUNT, bool PMASK, typename Next>
__device__ __forceinline__ void lkb_walk(const ScoreArgs<Real>& s, const LkbArgs<Real>& k, const LkbEval<Real>& ev,
                                         LkbWarp<Real, TAGGED>& q, LkbList<Real, TAGGED>& L, const LkbRows& a,
                                         Real cx, Real cy, Real cz, Real reach2, int n_cand, Next next,
                                         const Lkb4<Real> w, Real* e4, const LkbTagged<Real> tg) {
  const int lane = q.lane;
  const unsigned lemask = q.lt_mask | (1u << lane);
  const int nc1 = PMASK ? 0 : s.bt_n_conn[a.bt];
  const int rtf0 = lane < a.nocc ? s.hpacked[a.hb + lane].tf : 0;  // the first 32 rows
  int m = 0;  // atoms in the list
  for (int c0 = 0; c0 < n_cand; c0 += 32) {
    const LkbHit h = next(c0);
    if (COUNT) {
      q.n_bp += __popc(__ballot_sync(0xffffffffu, h.hit));
      const int pairs = !h.hit ? 0 : h.entry == -1 ? a.npol * a.nocc : a.npol * k.nocc[h.bt] + a.nocc * k.npol[h.bt];
      q.n_pairs += __reduce_add_sync(0xffffffffu, pairs);
    }
    const int n = h.hit ? k.nocc[h.bt] : 0;
    int inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    const int T = __shfl_sync(0xffffffffu, inc, 31);
    const int start = n > 0 ? inc - n : 0x7fffffff;
    const unsigned hm = __ballot_sync(0xffffffffu, n > 0);
    __syncwarp();
    if (n > 0) {
      const int slot = __popc(hm & q.lt_mask);
      L.hoff[slot] = h.hb - start;
      L.off[slot] = h.off;
      L.bt[slot] = h.bt;
      L.ent[slot] = h.entry;
      if (TAGGED) L.htag[slot] = h.tag;
    }
    __syncwarp();
    const bool final = c0 + 32 >= n_cand;
    int owned = 0;
    for (int k0 = 0; k0 < T || (final && m > 0); k0 += 32) {
      if (k0 < T) {
        // 32 atoms of the flat list: bit p of `word` set where a neighbour's
        // atoms begin at list position k0 + p
        const unsigned pos = (unsigned)(start - k0);
        const unsigned word = __reduce_or_sync(0xffffffffu, pos < 32u ? 1u << pos : 0u);
        const int own = max(owned + __popc(word & lemask) - 1, 0);
        owned += __popc(word);
        AtomRec<Real> o;
        o.x = o.y = o.z = Real(0);
        o.tf = 0;
        const bool valid = k0 + lane < T;
        if (valid) o = s.hpacked[L.hoff[own] + k0 + lane];
        const Real dx = o.x - cx, dy = o.y - cy, dz = o.z - cz;
        const bool keep = valid && dx * dx + dy * dy + dz * dz < reach2;
        const unsigned km = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          const int j = m + __popc(km & q.lt_mask);
          L.x[j] = o.x;
          L.y[j] = o.y;
          L.z[j] = o.z;
          L.tf[j] = o.tf;
          L.row[j] = L.off[own] + (o.tf & kHeavyAtom);
          L.par[j] = L.bt[own] * s.A + (o.tf & kHeavyAtom);
          L.entry[j] = L.ent[own];
          if (TAGGED) L.tag[j] = L.htag[own];
        }
        m += __popc(km);
        __syncwarp();
      }
      if (m < 32 && !(final && k0 + 32 >= T && m > 0)) continue;
      // the list's first 32 atoms against every row: the row polar and the
      // list's atom occluding, then the other way round; of a list of 16 or 8
      // atoms, an item's last, two or four lanes share one, each with every
      // second or fourth row
      const int shift = m > 16 ? 0 : (m > 8 ? 1 : 2), rep = 1 << shift;
      const int at_l = lane & ((32 >> shift) - 1), sub = lane >> (5 - shift);
      AtomRec<Real> o;
      o.x = L.x[at_l];
      o.y = L.y[at_l];
      o.z = L.z[at_l];
      o.tf = L.tf[at_l];
      const int entry = L.entry[at_l], ja = o.tf & kHeavyAtom;
      const bool valid = at_l < m;
      const bool special = valid && entry != -2;
      const bool any_special = __any_sync(0xffffffffu, special);
      for (int rt = 0; rt < a.nocc; rt += 32) {
        const int nr = min(32, a.nocc - rt);
        const int rtf = rt == 0 ? rtf0 : (lane < nr ? s.hpacked[a.hb + rt + lane].tf : 0);
        // bit i: row rt + i and this lane's atom are a pair in reach (near)
        // with weight 0.2 (four): no branch or vote in the rows' loads
        unsigned near = 0, four = 0;
        const unsigned mine = valid ? 0xffffffffu >> (32 - nr) : 0u;  // rows
#pragma unroll (GRAD ? 1 : 4)
        for (int i0 = 0; i0 < nr; i0 += rep) {
          const int i = i0 + sub;
          const AtomRec<Real> r = s.hpacked[a.hb + rt + min(i, nr - 1)];
          const Real dv[3] = {r.x - o.x, r.y - o.y, r.z - o.z};
          near |= (lkb_within(lkb_dot(dv, dv), k.max_dis) ? 1u : 0u) << i;
        }
        near &= mine;
        if (any_special) {
          unsigned out = 0;
          const uint2* masks = nullptr;  // of the word that holds this atom, by row atom
          int64_t stride = 1;
          if (special && entry == -1) {
            masks = s.imask + (int64_t)a.bt * s.A * s.n_iwords + (ja >> 5);
            stride = s.n_iwords;
          } else if (PMASK && special) {
            masks = s.pmask + s.cp_moff[entry] + (int64_t)(ja >> 5) * a.n_atoms;
          }
#pragma unroll (GRAD ? 1 : 4)
          for (int i0 = 0; i0 < nr; i0 += rep) {
            const int i = i0 + sub;
            const int ra = __shfl_sync(0xffffffffu, rtf, i) & kHeavyAtom;  // past nr: 0
            uint2 mk = make_uint2(0u, 0u);
            if (masks) mk = masks[ra * stride];
            out |= ((mk.x >> (ja & 31)) & 1u) << i;
            four |= ((mk.y >> (ja & 31)) & 1u) << i;
          }
          if (!PMASK) {
            // a count-pair partner: its atom's separation from each of the
            // rows' connections, a byte each, then row by row
            const bool partner = special && entry >= 0;
            unsigned far = 0x3f3f3f3fu;
            if (partner) {
              const int bt2 = (L.par[at_l] - ja) / s.A, nc2 = s.bt_n_conn[bt2];
              const uint8_t* seps = s.cp_seps + (int64_t)entry * 16;
              const uint32_t cj = load_cpd(s, bt2, nc2, ja);
              for (int u = 0; u < nc1; ++u) {
                int best = 63;
                for (int v = 0; v < nc2; ++v)
                  best = min(best, (int)seps[u * 4 + v] + (int)((cj >> (8 * v)) & 0xff));
                far = (far & ~(0xffu << (8 * u))) | ((unsigned)best << (8 * u));
              }
            }
            if (__any_sync(0xffffffffu, partner)) {
              const uint32_t c0 = lane < nr ? load_cpd(s, a.bt, nc1, rtf & kHeavyAtom) : 0u;
              for (int i0 = 0; i0 < nr; i0 += rep) {
                const int i = i0 + sub;
                const uint32_t ci = __shfl_sync(0xffffffffu, c0, i);
                int sep = 5;
                for (int u = 0; u < nc1; ++u)
                  sep = min(sep, (int)((ci >> (8 * u)) & 0xff) + (int)((far >> (8 * u)) & 0xff));
                if (partner) {
                  out |= (unsigned)(sep < 4) << i;
                  four |= (unsigned)(sep == 4) << i;
                }
              }
            }
          }
          near &= ~out;
        }
        // the pairs in either direction: the row polar and the list's atom
        // occluding, then the other way round; one of each lane at a time
        const unsigned polar_rows = __ballot_sync(0xffffffffu, rtf & kHeavyPolar);
        const unsigned bridge_rows = __ballot_sync(0xffffffffu, rtf & kHeavyBridges);
        unsigned there = near & polar_rows, back = (o.tf & kHeavyPolar) ? near : 0u;
        for (;;) {
          const bool act = (there | back) != 0, bk = there == 0;
          const int i = act ? __ffs(bk ? back : there) - 1 : 0;
          const bool bridged = bk ? (bridge_rows >> i) & 1u : (L.tf[at_l] & kHeavyBridges) != 0;
          const unsigned m1 = __ballot_sync(0xffffffffu, act && bridged);
          const unsigned m0 = __ballot_sync(0xffffffffu, act && !bridged);
          if ((m0 | m1) == 0) break;
          const int ra = __shfl_sync(0xffffffffu, rtf, i) & kHeavyAtom;
          if (act) {
            if (bk)
              back &= back - 1;
            else
              there &= there - 1;
            const int rr = a.off + ra, rpar = a.bt * s.A + ra, orow = L.row[at_l], opar = L.par[at_l];
            LkbQueue<TAGGED>& Q = q.qs[bridged ? 1 : 0];
            const int at = (bridged ? q.nq[1] : q.nq[0]) + __popc((bridged ? m1 : m0) & q.lt_mask);
            Q.rp[at] = bk ? orow : rr;
            Q.ro[at] = bk ? rr : orow;
            Q.pi[at] = bk ? opar : rpar;
            Q.oi[at] = bk ? rpar : opar;
            Q.sep[at] = (four >> i) & 1u ? 4 : 6;
            if (TAGGED) Q.tag[at] = L.tag[at_l];
          }
          q.nq[0] += __popc(m0);
          q.nq[1] += __popc(m1);
          if (COUNT) {
            q.n_eval += __popc(m0 | m1);
            q.n_bridge += __popc(m1);
          }
          lkb_pump<Real, GRAD, TAGGED>(ev, q, false, w, e4, tg);
        }
      }
      // the rest of the list to its front
      const int rest = m > 32 ? m - 32 : 0;
      __syncwarp();
      if (lane < rest) {
        L.x[lane] = L.x[32 + lane];
        L.y[lane] = L.y[32 + lane];
        L.z[lane] = L.z[32 + lane];
        L.tf[lane] = L.tf[32 + lane];
        L.row[lane] = L.row[32 + lane];
        L.par[lane] = L.par[32 + lane];
        L.entry[lane] = L.entry[32 + lane];
        if (TAGGED) L.tag[lane] = L.tag[32 + lane];
      }
      m = rest;
      __syncwarp();
    }
  }
}

// The count-pair table entry of block b2 in row i1 (cp_b2: the row's
// partners, one per lane), or -2.
template <typename Real>
__device__ __forceinline__ int lkb_entry(const ScoreArgs<Real>& s, int64_t i1, int ncp, int cp_b2, int b2) {
  int e = -2;
  for (int p = 0; p < ncp; ++p)
    if (__shfl_sync(0xffffffffu, cp_b2, p) == b2) e = (int)(i1 * CP_CAP + p);
  return e;
}

template <typename Real>
__device__ __forceinline__ LkbEval<Real> lkb_eval_of(const ScoreArgs<Real>& s, const LkbArgs<Real>& k) {
  LkbEval<Real> ev;
  ev.coords = s.coords;
  ev.waters = k.waters;
  ev.par = k.par;
  ev.dcoords = s.dcoords;
  ev.dwaters = k.dwaters_out;
  ev.vec_w = (reinterpret_cast<uintptr_t>(k.waters) & (4 * sizeof(Real) - 1)) == 0;
  ev.vec_dw = (reinterpret_cast<uintptr_t>(k.dwaters_out) & (4 * sizeof(Real) - 1)) == 0;
  ev.water_dist = k.water_dist;
  ev.hbond_dis = k.hbond_dis;
  ev.hbond_oh = k.hbond_oh;
  ev.hbond_h = k.hbond_h;
  ev.max_dis = k.max_dis;
  return ev;
}

template <typename Real, bool TAGGED>
__device__ __forceinline__ void lkb_flush_counts(const ScoreArgs<Real>& s, const LkbWarp<Real, TAGGED>& q) {
  if (s.counts && q.lane == 0) {
    if (q.n_bp) atomicAdd(&s.counts[0], q.n_bp);
    if (q.n_pairs) atomicAdd(&s.counts[1], q.n_pairs);
    if (q.n_bridge) atomicAdd(&s.counts[2], q.n_bridge);
    if (q.n_eval) atomicAdd(&s.counts[3], q.n_eval);
  }
}

// The pose op: the plan's work items (pose, b1, candidate blocks b2 >= b1),
// the neighbour rule as score_kernel applies it, then every polar /
// occluder pair of each neighbouring block pair.
// COUNT: the work counters (registers and instructions in the pair loop),
// compiled into a separate instantiation used on request
template <typename Real, bool GRAD, bool BLOCK_PAIR, bool COUNT>
__global__ void __launch_bounds__(256, lkb_min_ctas<Real, GRAD>) lkb_score_kernel(ScoreArgs<Real> s, LkbArgs<Real> k, int items_per_ticket) {
  if (s.done && *s.done) return;  // a speculative gradient was taken
  // [warp][plain, bridged]; block-pair mode tags queued pairs with their
  // block pair (p * B + b1) * B + b2
  __shared__ LkbQueue<BLOCK_PAIR> queues[LKB_MAX_WARPS][2];
  __shared__ LkbList<Real, BLOCK_PAIR> lists[LKB_MAX_WARPS];
  LkbWarp<Real, BLOCK_PAIR> q;
  q.lane = threadIdx.x & 31;
  q.qs = queues[threadIdx.x >> 5];
  q.lt_mask = (1u << q.lane) - 1u;
  q.nq[0] = q.nq[1] = 0;
  q.n_bp = q.n_pairs = q.n_bridge = q.n_eval = 0;
  const int lane = q.lane;
  const int64_t stride = (int64_t)s.P * s.B * s.B;
  const LkbEval<Real> ev = lkb_eval_of(s, k);
  LkbTagged<Real> tg;
  tg.energies = s.energies;
  tg.dTdV = s.dTdV;
  tg.n = stride;
  const Lkb4<Real> none = {{0, 0, 0, 0}};
  const int n_work = s.ticket[2];  // the plan's item count (a rebalance may split items)
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(s.ticket, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    const int it0 = t * items_per_ticket;
    if (it0 >= n_work) break;
    const int it1 = min(it0 + items_per_ticket, n_work);
    for (int item = it0; item < it1; ++item) {
      const long long t_item = COUNT ? clock64() : 0;  // item costs: the counting instantiation
      const int4 wi = s.work[item];
      const int p = wi.x, b1 = wi.y, cand0 = wi.z, cand1 = wi.w;
      const int i1 = p * s.B + b1;
      const int bt1 = s.blk_bt[i1];
      if (bt1 < 0) {
        if (s.item_cost && lane == 0) s.item_cost[item] = 0;
        continue;
      }
      const Quad<Real> sph1 = reinterpret_cast<const Quad<Real>*>(s.spheres)[i1];
      // the row's count-pair partners, one per lane
      const int ncp = s.cp_count[i1];
      const int cp_b2 = lane < ncp ? s.cp_b2[(int64_t)i1 * CP_CAP + lane] : -1;
      Lkb4<Real> w = {{0, 0, 0, 0}};
      if (GRAD && !BLOCK_PAIR)
        for (int c = 0; c < 4; ++c) w.v[c] = s.dTdV[(int64_t)c * s.P + p];
      Real acc[4] = {0, 0, 0, 0};
      const LkbRows rows = {bt1, s.blk_off[i1], k.hbase[i1], k.nocc[bt1], k.npol[bt1], s.bt_n_atoms[bt1]};
      const Real reach1 = sph1.d + k.max_dis;
      auto next = [&](int first) {
        const int b2 = cand0 + first + lane;
        LkbHit h = {false, -2, 0, 0, 0, 0};
        h.entry = lkb_entry(s, i1, ncp, cp_b2, b2);
        if (b2 < cand1) {
          const int i2 = p * s.B + b2;
          const int bt2 = s.blk_bt[i2];
          if (bt2 >= 0) {
            const Quad<Real> s2 = reinterpret_cast<const Quad<Real>*>(s.spheres)[i2];
            const Real dx = sub_rn(sph1.a, s2.a), dy = sub_rn(sph1.b, s2.b), dz = sub_rn(sph1.c, s2.c);
            const Real d2 = add_rn(add_rn(mul_rn(dx, dx), mul_rn(dy, dy)), mul_rn(dz, dz));
            const Real thr = add_rn(add_rn(sph1.d, s2.d), s.reach);
            h.hit = d2 < mul_rn(thr, thr);
            h.bt = bt2;
            h.off = s.blk_off[i2];
            h.hb = k.hbase[i2];
            if (BLOCK_PAIR) h.tag = (int)((int64_t)i1 * s.B + b2);
            if (b2 == b1) h.entry = -1;
          }
          if (s.nbr) s.nbr[(int64_t)i1 * s.B + b2] = h.hit ? 1 : 0;
        }
        return h;
      };
      lkb_walk<Real, GRAD, BLOCK_PAIR, COUNT, true>(s, k, ev, q, lists[threadIdx.x >> 5], rows, sph1.a, sph1.b,
                                                    sph1.c, reach1 * reach1 * Real(1.0001), cand1 - cand0, next,
                                                    BLOCK_PAIR ? none : w, acc, tg);
      if (!BLOCK_PAIR) lkb_pump<Real, GRAD, BLOCK_PAIR>(ev, q, true, w, acc, tg);
      // whole-pose energies (also in the adjoint when asked for: one pass
      // for energy and gradient)
      if (!BLOCK_PAIR && s.energies)
        for (int c = 0; c < 4; ++c) {
          const Real v = warp_sum(acc[c]);
          if (lane == 0 && v != Real(0)) atomicAdd(&s.energies[(int64_t)c * s.P + p], v);
        }
      // the item's cost, for ordering the work longest-first
      if (COUNT && s.item_cost && lane == 0)
        s.item_cost[item] = (int)min((clock64() - t_item) >> 4, (long long)0x7fffffff);
    }
  }
  if (BLOCK_PAIR) {
    Real unused[4] = {0, 0, 0, 0};  // tagged entries add their energies to their rows
    lkb_pump<Real, GRAD, BLOCK_PAIR>(ev, q, true, none, unused, tg);
  }
  lkb_flush_counts(s, q);
}

// The rotamer op: work items (rot1, first rot2, n rot2, first pair) from
// the rotamer dispatch; every polar / occluder pair of rot1 against each
// rot2 (itself on the diagonal), energies per dispatched pair
// (energies[t * n_pairs + d], added by atomics), the adjoint under
// dTdV[t * n_pairs + d].  Queued pairs carry d, so the queues fill across
// rotamer pairs and items (a rotamer pair has few pairs in reach).
template <typename Real, bool GRAD, bool COUNT>
__global__ void __launch_bounds__(256, lkb_min_ctas<Real, GRAD>)
    lkb_rotamer_kernel(ScoreArgs<Real> s, LkbArgs<Real> k, RotArgs ra, const Real* rot_spheres) {
  __shared__ LkbQueue<true> queues[LKB_MAX_WARPS][2];
  __shared__ LkbList<Real, true> lists[LKB_MAX_WARPS];
  LkbWarp<Real, true> q;
  q.lane = threadIdx.x & 31;
  q.qs = queues[threadIdx.x >> 5];
  q.lt_mask = (1u << q.lane) - 1u;
  q.nq[0] = q.nq[1] = 0;
  q.n_bp = q.n_pairs = q.n_bridge = q.n_eval = 0;
  const int lane = q.lane;
  const LkbEval<Real> ev = lkb_eval_of(s, k);
  LkbTagged<Real> tg;
  tg.energies = s.energies;
  tg.dTdV = s.dTdV;
  tg.n = ra.n_pairs;
  const Lkb4<Real> none = {{0, 0, 0, 0}};
  Real unused[4] = {0, 0, 0, 0};  // tagged entries add their energies to their rows
  for (;;) {
    int it = 0;
    if (lane == 0) it = atomicAdd(s.ticket, 1);
    it = __shfl_sync(0xffffffffu, it, 0);
    if (it >= ra.n_items) break;
    const int4 item = ra.items[it];
    const int rot1 = item.x, rot2_first = item.y, n_rot2 = item.z;
    const long long pair_first = item.w;
    const int p = ra.rot_pose[rot1], b1 = ra.rot_block[rot1];
    const int64_t i1 = (int64_t)p * s.B + b1;
    const int bt1 = ra.rot_bt[rot1];
    const LkbRows rows = {bt1, ra.rot_off[rot1], k.hbase[rot1], k.nocc[bt1], k.npol[bt1], s.bt_n_atoms[bt1]};
    // b2 and its count-pair entry are the same for every rot2 of the item
    const int ncp = s.cp_count[i1];
    const int cp_b2 = lane < ncp ? s.cp_b2[i1 * CP_CAP + lane] : -1;
    const int b2 = n_rot2 > 0 ? ra.rot_block[rot2_first] : b1;
    const int entry = lkb_entry(s, i1, b2 != b1 ? ncp : 0, cp_b2, b2);
    const Quad<Real> sp1 = reinterpret_cast<const Quad<Real>*>(rot_spheres)[rot1];
    const Real reach1 = sp1.d + k.max_dis;
    auto next = [&](int first) {
      const int j = first + lane;
      LkbHit h = {false, entry, 0, 0, 0, 0};
      if (j < n_rot2) {
        const int rot2 = rot2_first + j;
        const bool self = rot2 == rot1;
        // no atom pair of two rotamers whose bounding spheres are farther
        // apart than max_dis (with a margin far above rounding) is in reach:
        // their energies are zero
        const Quad<Real> q2 = reinterpret_cast<const Quad<Real>*>(rot_spheres)[rot2];
        const Real dx = sp1.a - q2.a, dy = sp1.b - q2.b, dz = sp1.c - q2.c;
        const Real thr = sp1.d + q2.d + k.max_dis + Real(0.01);
        h.hit = self || !(dx * dx + dy * dy + dz * dz > thr * thr);
        if (self) h.entry = -1;
        h.bt = ra.rot_bt[rot2];
        h.off = ra.rot_off[rot2];
        h.hb = k.hbase[rot2];
        h.tag = (int)(pair_first + j);
      }
      return h;
    };
    lkb_walk<Real, GRAD, true, COUNT, false>(s, k, ev, q, lists[threadIdx.x >> 5], rows, sp1.a, sp1.b, sp1.c,
                                             reach1 * reach1 * Real(1.0001), n_rot2, next, none, unused, tg);
  }
  // entries carry their pair: the queues drain across items, once at the end
  lkb_pump<Real, GRAD, true>(ev, q, true, none, unused, tg);
  lkb_flush_counts(s, q);
}
