// The atom-pair engine of the LJ/LK and elec kernels: one warp scores the
// atoms of one block (or rotamer) against those of its neighbours.
// Included by ljlk.cu inside namespace tmol_b200, after ScoreArgs.
//
// A warp works in groups.  The rows are up to 32 atoms of block b1, one per
// lane, in registers; side 1 is a list of up to M1 neighbouring atoms in the
// warp's shared-memory slab.  A group goes through three phases:
//   1. screening: side 1 comes in words of up to 32 atoms.  Every lane tests
//      its row against a word's atoms (broadcast, four at a time, packed
//      pairs of float32 operations) and shifts the sign bits of d^2 - max^2
//      and d^2 - far^2 into two masks: no compare, vote or branch per pair.
//      Bonded neighbours and b1 itself have exclusion masks beside them.
//   2. emission: each (row, word) writes its surviving pairs into a queue of
//      16-bit entries, in three classes: far (both potentials are the cubic
//      fade to zero), near without a heavy pair (LJ alone) and near heavy.
//   3. evaluation, class by class: every lane takes an equal stretch of
//      consecutive entries.  Lanes of a step run the same code, a stretch
//      stays on one or two rows (their atom and force stay in registers), and
//      the side-1 forces go out as 16-byte vector reductions into a padded
//      gradient buffer.  Energies of pairs (blocks, rotamers) are evaluated a
//      window of entries at a time and added up pair by pair.
//
// What bounds it: latency, at 20 warps per SM (59% of the issue slots are
// used, the FMA pipes 26%, DRAM 1%; 64 x 150 residues, energy + gradient, 129
// us and 82 M warp instructions, where warps that listed pairs and summed both
// atoms' forces in shared memory took 302 us and 137 M).  So the loads an item
// starts from go out together, a whole list of neighbouring atoms is in flight
// at once (cp.async into side 1, culled in place), and forces leave the SM
// without being waited for: shared-memory float atomics are compare-and-swap
// loops here (64 x 150 residues, energy + gradient: 185 us with the side-1
// forces summed in shared memory, 138 us without); a red.global.add.v4.f32 is
// one instruction that nothing waits for.

constexpr int M1 = 160;  // side-1 atoms of a group (< 256: 8-bit index)
constexpr int MAXW = 9;  // words of a group; odd: the mask arrays' row stride has no bank conflicts
constexpr int MAXSP = 4; // words with exclusion masks
// Warps per CTA and SM.  The engine waits on memory more than it issues, so
// warps count for more than registers or a longer side 1: 64 x 150 residues,
// energy + gradient, 16 warps of 128 registers take 144 us with M1 = 224 and
// 142 us with 160; 20 warps of 96 registers 130 us with 160 and with 128
// (before forces were split).
constexpr int PAIR_WARPS = 20;
// A whole-pose group holds up to MAXSP words with masks and the flat list's
// M1 / 32 beside them (its room test leaves those out), and a queue entry has
// 8 bits for the atom.
static_assert(M1 % 32 == 0 && M1 / 32 + MAXSP <= MAXW && M1 < 256, "a group's words and atoms");
constexpr int kTfHeavy = 256;

// One atom: coordinates and either the compact atom type | heavy << 8
// (LJ/LK) or the partial charge (elec).
template <typename Real>
struct alignas(16) AtomRec {
  Real x, y, z;
  union {
    int tf;
    Real q;
  };
};

// Queue entry: side-1 atom (bits 0-7), row (8-12), count-pair weight 0.2 (13).
// The queue lives where the screening coordinates were: they are read out
// before the first entry is written.  A single word (32 x 32 pairs) always
// fits; a group with more pairs than the queue holds goes word by word.
template <typename Real>
struct Slab {
  static constexpr int QCAP = 3 * M1 * sizeof(Real) / 2 < 1024 ? 1024 : 3 * M1 * sizeof(Real) / 2;
  static_assert(QCAP >= 32 * 32, "a word's pairs");
  AtomRec<Real> at[M1];
  union {
    struct {
      Real x[M1], y[M1], z[M1];
    } c;
    uint16_t queue[QCAP];
  };
  uint32_t far[32 * MAXW], near[32 * MAXW];  // [row][word]
  uint2 smask[MAXSP][32];                            // per row: excluded, weight 0.2
  AtomRec<Real> row[32];
  long long out[MAXW];  // pair mode: the word's energy entry
  int desc[MAXW];       // base | atoms << 8 | (mask + 1) << 16
  uint32_t heavy[MAXW];
  uint8_t slot[M1];  // pair mode: the atom's word
  // last, and next to each other: pair energies use their place (PairSums)
  int gidx[M1];  // global atom index (gradients)
  int hoff[32];  // pose mode: the flat list's hits
};

// Pair energies (no gradient): the energies of up to EWIN queue entries, from
// which each word's are added in the order of its entries, and where each
// word's entries begin in each class.  In float the window lies on the index
// lists that only gradients and pose mode have; with the 448 bytes that it
// takes beyond the slab, 20 warps stay within 196 KB of shared memory, which
// leaves L1 60 KB.
constexpr int EWIN = 96;
template <typename Real>
struct PairSums {
  static constexpr size_t at = sizeof(Real) == 4 ? offsetof(Slab<Real>, gidx) : sizeof(Slab<Real>);
  Real e[3][EWIN];
  uint16_t first[3][MAXW + 1];
  uint16_t pad[2];
};
static_assert(PairSums<float>::at % 16 == 0 && sizeof(PairSums<float>) % 16 == 0 && sizeof(PairSums<double>) % 16 == 0,
              "a warp's slab keeps its alignment");
static_assert(offsetof(Slab<float>, gidx) + (M1 + 32) * sizeof(int) == sizeof(Slab<float>),
              "the float sums lie on the slab's last members");

// Bytes of a warp's slab; sums: of one that adds up pair energies.
template <typename Real>
__host__ __device__ constexpr size_t slab_bytes(bool sums) {
  return sums ? PairSums<Real>::at + sizeof(PairSums<Real>) : sizeof(Slab<Real>);
}
template <typename Real>
__device__ __forceinline__ PairSums<Real>& pair_sums(Slab<Real>& w) {
  return *reinterpret_cast<PairSums<Real>*>(reinterpret_cast<char*>(&w) + PairSums<Real>::at);
}

template <typename Real>
__device__ __forceinline__ Real warp_sum(Real v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <typename Real>
struct E3 {
  Real atr, rep, lk;
};

// What evaluating a pair needs beside the slab.
template <typename Real>
struct EvalCtx {
  const Quad<Real>* lj;   // [2][ntp * ntp] LJ groups
  const LKRecord<Real>* lk;
  const Quad<Real>* far;  // [ntp * ntp] fade-out knots of both potentials
  const Real* elec_k;
  int ntp;
  Real max2, far2;        // squares of the cutoff and of the far class's start
  Real far_dmin, far_first, inv_hf;
  Real wt0, wt1, wt2;     // gradient weights of the three terms (elec: wt0)
  Real grid;              // force_grid_of them
  Real* g;                // padded gradient [n_atoms][GRAD_STRIDE]
  int64_t row0;           // global atom index of row 0
  Real* energies;         // pair mode: [n_terms][stride]
  const Real* dTdV;       // pair mode: the same shape
  int64_t stride;
};

// Adds a force to an atom's padded gradient: GRAD_STRIDE values, two groups
// (x, y, z, -) whose sum is the gradient.  The first group takes multiples of
// 2^-6 kcal/mol/A, whose float32 sums are exact (below 2^18) and so the same
// in any order; what remains of a force goes to the second, whose sums stay
// small.  A single float32 sum of forty signed terms in no fixed order, where
// clashes of 10^3 kcal/mol/A nearly cancel, differs by 3e-4 from call to call.
// These figures are for forces of up to 2^16 under weights of about one; the
// grid scales with the power of two of the largest weight, so that they hold
// relative to the weights whatever the caller's loss is multiplied by.
// (Larger forces, and weights of unlike size on one atom, are summed right but
// on coarser or several grids.)
// SMALL: a force of the far class (about one, weighted alike), to the second
// group alone.
constexpr int GRAD_STRIDE = 8;

// What force_grid rounds with: 1.5 x 2^17 (float32 spacing 2^-6) times the
// power of two at or below the largest weight's magnitude m.
__device__ __forceinline__ float force_grid_of(float m) {
  return 1.5f * 131072.0f * __uint_as_float(__float_as_uint(fminf(m, 0x1p100f)) & 0x7f800000u);
}
__device__ __forceinline__ double force_grid_of(double) { return 0.0; }  // not split

__device__ __forceinline__ void red4(float* g, float x, float y, float z) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(g), "f"(x), "f"(y), "f"(z), "f"(0.0f)
               : "memory");
}
// The part of x on the grid; none of an infinite x, whose remainder would be a NaN.
__device__ __forceinline__ float on_grid(float x, float grid) {
  const float h = __fsub_rn(__fadd_rn(x, grid), grid);
  return fabsf(x) < 0x1p127f ? h : 0.0f;
}
template <bool SMALL = false>
__device__ __forceinline__ void add_force(float* g, float grid, float x, float y, float z) {
  if (SMALL) {
    red4(g + 4, x, y, z);
    return;
  }
  const float hx = on_grid(x, grid), hy = on_grid(y, grid), hz = on_grid(z, grid);
  if (hx != 0.0f || hy != 0.0f || hz != 0.0f) red4(g, hx, hy, hz);
  red4(g + 4, __fsub_rn(x, hx), __fsub_rn(y, hy), __fsub_rn(z, hz));
}
template <bool SMALL = false>
__device__ __forceinline__ void add_force(double* g, double, double x, double y, double z) {
  atomicAdd(g, x);
  atomicAdd(g + 1, y);
  atomicAdd(g + 2, z);
}

// One atom record from global to shared memory, without a register.
template <typename Real>
__device__ __forceinline__ void copy_async(AtomRec<Real>* dst, const AtomRec<Real>* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
#pragma unroll
  for (int k = 0; k < (int)sizeof(AtomRec<Real>); k += 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + k), "l"((const char*)src + k) : "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Packed pairs of float32 operations.
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b,
                                                   unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// Screens one row against side-1 atoms [base, base + cnt): bit k of `in`
// (d^2 < max2) and `near` (d^2 < far2).  Bits at and above cnt are undefined.
struct RowTest {
  unsigned in, near;
};

__device__ __forceinline__ RowTest test_row(const Slab<float>& w, int base, int cnt, float x, float y, float z,
                                            float max2, float far2) {
  const unsigned long long nx = pack2(-x, -x), ny = pack2(-y, -y), nz = pack2(-z, -z);
  const unsigned long long cm = pack2(-max2, -max2), gap = pack2(max2 - far2, max2 - far2);
  unsigned in = 0, near = 0;
  for (int j = (cnt - 1) & ~3; j >= 0; j -= 4) {
    const float4 X = *reinterpret_cast<const float4*>(w.c.x + base + j);
    const float4 Y = *reinterpret_cast<const float4*>(w.c.y + base + j);
    const float4 Z = *reinterpret_cast<const float4*>(w.c.z + base + j);
    const unsigned long long dxa = add2(pack2(X.x, X.y), nx), dxb = add2(pack2(X.z, X.w), nx);
    const unsigned long long dya = add2(pack2(Y.x, Y.y), ny), dyb = add2(pack2(Y.z, Y.w), ny);
    const unsigned long long dza = add2(pack2(Z.x, Z.y), nz), dzb = add2(pack2(Z.z, Z.w), nz);
    const unsigned long long ta = fma2(dza, dza, fma2(dya, dya, fma2(dxa, dxa, cm)));
    const unsigned long long tb = fma2(dzb, dzb, fma2(dyb, dyb, fma2(dxb, dxb, cm)));
    const unsigned long long ga = add2(ta, gap), gb = add2(tb, gap);
    float t0, t1, t2, t3, g0, g1, g2, g3;
    unpack2(ta, t0, t1);
    unpack2(tb, t2, t3);
    unpack2(ga, g0, g1);
    unpack2(gb, g2, g3);
    // the last atom first: after the loop atom k's sign is bit k
    in = __funnelshift_l(__float_as_uint(t3), in, 1);
    in = __funnelshift_l(__float_as_uint(t2), in, 1);
    in = __funnelshift_l(__float_as_uint(t1), in, 1);
    in = __funnelshift_l(__float_as_uint(t0), in, 1);
    near = __funnelshift_l(__float_as_uint(g3), near, 1);
    near = __funnelshift_l(__float_as_uint(g2), near, 1);
    near = __funnelshift_l(__float_as_uint(g1), near, 1);
    near = __funnelshift_l(__float_as_uint(g0), near, 1);
  }
  return RowTest{in, near};
}

__device__ __forceinline__ RowTest test_row(const Slab<double>& w, int base, int cnt, double x, double y, double z,
                                            double max2, double far2) {
  unsigned in = 0, near = 0;
  for (int j = cnt - 1; j >= 0; --j) {
    const double dx = w.c.x[base + j] - x, dy = w.c.y[base + j] - y, dz = w.c.z[base + j] - z;
    const double d2 = dx * dx + dy * dy + dz * dz;
    in = (in << 1) | (d2 < max2 ? 1u : 0u);
    near = (near << 1) | (d2 < far2 ? 1u : 0u);
  }
  return RowTest{in, near};
}

enum PairClass : int { kFar = 0, kNear = 1, kNearHeavy = 2 };

template <typename Real, int TERM>
__device__ __forceinline__ Real grid_of_weights(Real wt0, Real wt1, Real wt2) {
  return force_grid_of(TERM == kTermElec ? fabs(wt0) : fmax(fabs(wt0), fmax(fabs(wt1), fabs(wt2))));
}

// One pair of a class: its energies, weighted by its count-pair weight wcp,
// and the force f (a - b) on a, (weighted dE/dd) / d.
template <typename Real>
struct PairTerms {
  Real e0, e1, e2, f;
};

template <typename Real, bool GRAD, int TERM, int CLS>
__device__ __forceinline__ PairTerms<Real> eval_pair(const EvalCtx<Real>& c, const ElecK<Real>& K,
                                                     const AtomRec<Real>& a, const AtomRec<Real>& b, Real dx, Real dy,
                                                     Real dz, Real wcp, Real wt0, Real wt1, Real wt2) {
  PairTerms<Real> p = {0, 0, 0, 0};
  const Real d2 = dx * dx + dy * dy + dz * dz;
  // coincident atoms (d2 = 0) take the linear LJ, flat LK and flat elec
  // regions, which never use inv_d, and add no force
  const Real inv_d = inv_sqrt(d2);
  const Real d = CLS == kFar || d2 > Real(0) ? d2 * inv_d : Real(0);
  if (TERM == kTermElec) {
    const Real wq = wcp * a.q * b.q;
    Real v, dv = 0;
    if (CLS == kFar) {
      const Real t = (d - K.hi_start) * K.inv_hi_w;
      v = K.hi[0] + t * (K.hi[1] + t * (K.hi[2] + t * K.hi[3]));
      if (GRAD) dv = (K.hi[1] + t * (Real(2) * K.hi[2] + Real(3) * t * K.hi[3])) * K.inv_hi_w;
    } else {
      elec_eval<Real, GRAD>(d, K, v, dv);
    }
    p.e0 = wq * v;
    if (GRAD) p.f = wq * wt0 * dv * inv_d;
  } else {
    const int tp = (a.tf & 0xff) * c.ntp + (b.tf & 0xff);
    if (CLS == kFar) {
      // both potentials fade on the same interval: a cubic from value V
      // and (interval-scaled) slope D to zero is V A(t) + D B(t), with
      // A = (1 - t)^2 (1 + 2 t), B = t (1 - t)^2
      const Quad<Real> k = c.far[tp];  // LJ value, slope; LK value, slope
      const Real t = (d - c.far_dmin) * c.inv_hf;
      const Real u = Real(1) - t;
      const Real uu = u * u;
      const Real A = uu + Real(2) * t * uu, B = t * uu;
      p.e0 = wcp * (k.a * A + k.b * B);
      p.e2 = wcp * (k.c * A + k.d * B);
      if (GRAD) {
        const Real dA = Real(-6) * t * u, dB = u - Real(3) * t * u;
        const Real V = wt0 * k.a + wt2 * k.c, D = wt0 * k.b + wt2 * k.d;
        p.f = wcp * c.inv_hf * inv_d * (V * dA + D * dB);
      }
    } else {
      Real atr, rep, datr, drep;
      lj_eval<Real, GRAD>(d, inv_d, c.lj + tp, c.lj + c.ntp * c.ntp + tp, atr, rep, datr, drep);
      p.e0 = wcp * atr;
      p.e1 = wcp * rep;
      Real dE = wt0 * datr + wt1 * drep;
      if (CLS == kNearHeavy) {
        Real lk, dlk;
        lk_eval<Real, GRAD>(d, inv_d, c.lk + tp, c.far_dmin, c.far_first, c.inv_hf, lk, dlk);
        p.e2 = wcp * lk;
        dE += wt2 * dlk;
      }
      if (GRAD) p.f = wcp * dE * inv_d;
    }
  }
  if (GRAD && CLS != kFar && d == Real(0)) p.f = 0;
  return p;
}

// Evaluates queue entries [q0, q0 + n) of one class.  Every lane takes a
// stretch of S consecutive entries (S kept off multiples of four, whose
// 16-bit stride would put the lanes' reads on the same banks).
template <typename Real, bool GRAD, bool PAIR, int TERM, int CLS>
__device__ __forceinline__ void eval_class(const EvalCtx<Real>& c, const Slab<Real>& w, int q0, int n, int lane,
                                           E3<Real>& acc) {
  static_assert(GRAD || !PAIR, "pair energies: sum_class");
  if (n == 0) return;
  int S = (n + 31) >> 5;
  if ((S & 3) == 0) ++S;
  const int cnt = min(S, n - lane * S);
  const uint16_t* q = w.queue + q0 + lane * S;
  int row = -1, slot = -1;
  AtomRec<Real> a;
  a.x = a.y = a.z = Real(0);
  a.tf = 0;
  Real fx = 0, fy = 0, fz = 0;
  Real wt0 = c.wt0, wt1 = c.wt1, wt2 = c.wt2, grid = c.grid;
  ElecK<Real> K;
  if (TERM == kTermElec) K = load_elec_k(c.elec_k);
  for (int s = 0; s < cnt; ++s) {
    const int e = q[s];
    const int j = e & 255, r = (e >> 8) & 31;
    if (r != row) {
      if (GRAD && row >= 0) {
        add_force<CLS == kFar>(c.g + GRAD_STRIDE * (c.row0 + row), grid, fx, fy, fz);
        fx = fy = fz = 0;
      }
      row = r;
      a = w.row[r];
    }
    if (PAIR) {
      const int sl = w.slot[j];
      if (sl != slot) {
        slot = sl;
        const Real* wt = c.dTdV + w.out[sl];
        wt0 = wt[0];
        if (TERM == kTermLJLK) {
          wt1 = wt[c.stride];
          wt2 = wt[2 * c.stride];
        }
        grid = grid_of_weights<Real, TERM>(wt0, wt1, wt2);
      }
    }
    const AtomRec<Real> b = w.at[j];
    const Real dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
    const Real wcp = (e >> 13) ? Real(0.2) : Real(1);
    const PairTerms<Real> p = eval_pair<Real, GRAD, TERM, CLS>(c, K, a, b, dx, dy, dz, wcp, wt0, wt1, wt2);
    if (!PAIR) {
      acc.atr += p.e0;
      acc.rep += p.e1;
      acc.lk += p.e2;
    }
    if (GRAD) {
      const Real px = p.f * dx, py = p.f * dy, pz = p.f * dz;
      fx += px;
      fy += py;
      fz += pz;
      add_force<CLS == kFar>(c.g + GRAD_STRIDE * (int64_t)w.gidx[j], grid, -px, -py, -pz);
    }
  }
  if (GRAD && row >= 0) add_force<CLS == kFar>(c.g + GRAD_STRIDE * (c.row0 + row), grid, fx, fy, fz);
}

// Pair energies: the lanes evaluate a window of a class's entries, then the
// lane of each word (k) and term (t) adds up the word's, one after the other,
// to v.  So a pair's energy is the same bits in every call, whichever pairs
// share its group.  (A sum per lane, added by an atomic a lane, is not;
// rotamers of 16 x 150 residues take 8.54 ms so and 8.44 ms with the window.
// A sum per row and word, each held by one lane, is, but takes 12.1 ms: a class
// of a group has two or three entries a lane, and whole rows balance badly.)
template <typename Real, int TERM, int CLS>
__device__ __forceinline__ void sum_class(const EvalCtx<Real>& c, Slab<Real>& w, int q0, int n, int lane, int k, int t,
                                          Real& v) {
  PairSums<Real>& ps = pair_sums(w);
  ElecK<Real> K;
  if (TERM == kTermElec) K = load_elec_k(c.elec_k);
  const bool adds = k >= 0 && !(CLS == kFar && t == 1) && !(CLS == kNear && t == 2);
  const int first = adds ? ps.first[CLS][k] : 0, last = adds ? ps.first[CLS][k + 1] : 0;
  for (int base = 0; base < n; base += EWIN) {
    const int m = min(EWIN, n - base);
    for (int i = lane; i < m; i += 32) {
      const int e = w.queue[q0 + base + i];
      const AtomRec<Real> a = w.row[(e >> 8) & 31], b = w.at[e & 255];
      const Real wcp = (e >> 13) ? Real(0.2) : Real(1);
      const PairTerms<Real> p = eval_pair<Real, false, TERM, CLS>(c, K, a, b, a.x - b.x, a.y - b.y, a.z - b.z, wcp,
                                                                  Real(0), Real(0), Real(0));
      ps.e[0][i] = p.e0;
      if (TERM == kTermLJLK && CLS != kFar) ps.e[1][i] = p.e1;
      if (TERM == kTermLJLK && CLS != kNear) ps.e[2][i] = p.e2;
    }
    __syncwarp();
    const int end = min(last - base, m);
    for (int i = max(first - base, 0); i < end; ++i) v += ps.e[t][i];
    __syncwarp();
  }
}

// Screens, queues and evaluates the group's words [0, nw) against rows
// [0, c1) (this lane's row at (rx, ry, rz)).  counts: pairs in reach, and
// heavy ones among them.
template <typename Real, bool GRAD, bool PAIR, int TERM, bool COUNT>
__device__ __forceinline__ void process_group(const EvalCtx<Real>& c, Slab<Real>& w, int nw, int c1, Real rx,
                                              Real ry, Real rz, unsigned heavy_rows, int lane, E3<Real>& acc,
                                              long long* counts) {
  __syncwarp();
  const bool hrow = (heavy_rows >> lane) & 1u;
  int n_far = 0, n_near = 0, n_heavy = 0;
  for (int k = 0; k < nw; ++k) {
    const int d = w.desc[k];
    const int base = d & 255, cnt = (d >> 8) & 63, sp = (d >> 16) - 1;
    const RowTest t = test_row(w, base, cnt, rx, ry, rz, c.max2, c.far2);
    unsigned live = lane < c1 ? 0xffffffffu >> (32 - cnt) : 0u;
    if (sp >= 0) live &= ~w.smask[sp][lane].x;
    const unsigned in = t.in & live;
    const unsigned fm = in & ~t.near, nm = in & t.near;
    w.far[lane * MAXW + k] = fm;
    w.near[lane * MAXW + k] = nm;
    n_far += __popc(fm);
    n_near += __popc(nm);
    if (TERM == kTermLJLK) {
      const unsigned hw = __ballot_sync(0xffffffffu, lane < cnt && (w.at[base + (lane < cnt ? lane : 0)].tf & kTfHeavy));
      if (lane == 0) w.heavy[k] = hw;
      if (hrow) n_heavy += __popc(nm & hw);
      if (COUNT && hrow) counts[1] += __popc(in & hw);
    }
  }
  __syncwarp();
  n_far = __reduce_add_sync(0xffffffffu, n_far);
  n_near = __reduce_add_sync(0xffffffffu, n_near);
  n_heavy = TERM == kTermLJLK ? __reduce_add_sync(0xffffffffu, n_heavy) : 0;
  if (COUNT && lane == 0) counts[0] += n_far + n_near;
  const bool whole = n_far + n_near <= Slab<Real>::QCAP;
  for (int ka = 0; ka < nw;) {
    int kb = nw;
    if (!whole) {
      kb = ka + 1;
      const unsigned nm = w.near[lane * MAXW + ka];
      n_far = __reduce_add_sync(0xffffffffu, __popc(w.far[lane * MAXW + ka]));
      n_near = __reduce_add_sync(0xffffffffu, __popc(nm));
      n_heavy = TERM == kTermLJLK ? __reduce_add_sync(0xffffffffu, hrow ? __popc(nm & w.heavy[ka]) : 0) : 0;
    }
    const int n_light = n_near - n_heavy;
    // emission: unit u is one (row, word); rows outermost, or words in pair
    // mode, so that a lane's stretch keeps its row (or energy entry)
    const int nwr = kb - ka, nu = nwr * c1;
    const int div = PAIR ? c1 : nwr;
    const int inv = 65536 / div + 1;  // u / div is exact for u <= 9 * 32
    int of = 0, ol = n_far, oh = n_far + n_light;
    for (int u0 = 0; u0 < nu; u0 += 32) {
      const int u = u0 + lane;
      unsigned F = 0, L = 0, H = 0, w02 = 0;
      int eb = 0, begins = -1;
      if (u < nu) {
        const int qd = (u * inv) >> 16, rem = u - qd * div;
        const int r = PAIR ? rem : qd, k = ka + (PAIR ? qd : rem);
        if (PAIR && rem == 0) begins = qd;
        F = w.far[r * MAXW + k];
        L = w.near[r * MAXW + k];
        if (TERM == kTermLJLK && ((heavy_rows >> r) & 1u)) {
          H = L & w.heavy[k];
          L &= ~H;
        }
        const int d = w.desc[k];
        eb = (r << 8) | (d & 255);
        const int sp = (d >> 16) - 1;
        if (sp >= 0) w02 = w.smask[sp][r].y;
      }
      const int mine = __popc(F) | (__popc(L) << 16), mine_h = __popc(H);
      int inc = mine, inc_h = mine_h;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        const int th = TERM == kTermLJLK ? __shfl_up_sync(0xffffffffu, inc_h, o) : 0;
        if (lane >= o) {
          inc += t;
          inc_h += th;
        }
      }
      const int tot = __shfl_sync(0xffffffffu, inc, 31);
      const int tot_h = TERM == kTermLJLK ? __shfl_sync(0xffffffffu, inc_h, 31) : 0;
      if (PAIR && !GRAD && begins >= 0) {
        PairSums<Real>& ps = pair_sums(w);
        ps.first[kFar][begins] = (uint16_t)(of + ((inc - mine) & 0xffff));
        ps.first[kNear][begins] = (uint16_t)(ol - n_far + ((inc - mine) >> 16));
        ps.first[kNearHeavy][begins] = (uint16_t)(oh - n_far - n_light + inc_h - mine_h);
      }
      uint16_t* qf = w.queue + of + ((inc - mine) & 0xffff);
      uint16_t* ql = w.queue + ol + ((inc - mine) >> 16);
      uint16_t* qh = w.queue + oh + (inc_h - mine_h);
      for (; F; F &= F - 1) {
        const int b = __ffs(F) - 1;
        *qf++ = (uint16_t)(eb + b + (((w02 >> b) & 1u) << 13));
      }
      for (; L; L &= L - 1) {
        const int b = __ffs(L) - 1;
        *ql++ = (uint16_t)(eb + b + (((w02 >> b) & 1u) << 13));
      }
      if (TERM == kTermLJLK)
        for (; H; H &= H - 1) {
          const int b = __ffs(H) - 1;
          *qh++ = (uint16_t)(eb + b + (((w02 >> b) & 1u) << 13));
        }
      of += tot & 0xffff;
      ol += tot >> 16;
      oh += tot_h;
    }
    if (PAIR && !GRAD && lane == 0) {
      PairSums<Real>& ps = pair_sums(w);
      ps.first[kFar][nwr] = (uint16_t)n_far;
      ps.first[kNear][nwr] = (uint16_t)n_light;
      ps.first[kNearHeavy][nwr] = (uint16_t)n_heavy;
    }
    __syncwarp();
    if constexpr (PAIR && !GRAD) {
      const int t = lane / MAXW, kw = lane % MAXW, k = kw < nwr && t < (TERM == kTermLJLK ? 3 : 1) ? kw : -1;
      Real v = 0;
      sum_class<Real, TERM, kFar>(c, w, 0, n_far, lane, k, t, v);
      sum_class<Real, TERM, kNear>(c, w, n_far, n_light, lane, k, t, v);
      if (TERM == kTermLJLK) sum_class<Real, TERM, kNearHeavy>(c, w, n_far + n_light, n_heavy, lane, k, t, v);
      // a pair's words are next to each other and go out one after the other
      const long long o = k >= 0 ? w.out[ka + k] : 0;
      int nth = 0;
      while (nth < k && w.out[ka + k - nth - 1] == o) ++nth;
      const int most = __reduce_max_sync(0xffffffffu, nth);
      for (int p = 0; p <= most; ++p) {
        if (p == nth && v != Real(0)) atomicAdd(c.energies + t * c.stride + o, v);
        __syncwarp();
      }
    } else {
      eval_class<Real, GRAD, PAIR, TERM, kFar>(c, w, 0, n_far, lane, acc);
      eval_class<Real, GRAD, PAIR, TERM, kNear>(c, w, n_far, n_light, lane, acc);
      if (TERM == kTermLJLK)
        eval_class<Real, GRAD, PAIR, TERM, kNearHeavy>(c, w, n_far + n_light, n_heavy, lane, acc);
    }
    __syncwarp();
    ka = kb;
  }
}

template <typename Real>
__device__ __forceinline__ uint32_t load_cpd(const ScoreArgs<Real>& s, int bt, int nconn, int at) {
  uint32_t v = 0x06060606u;
  for (int k = 0; k < nconn; ++k) {
    uint32_t d = s.bt_conn_pd[((int64_t)bt * s.C + k) * s.A + at];
    v = (v & ~(0xffu << (8 * k))) | (d << (8 * k));
  }
  return v;
}

template <typename Real>
__device__ __forceinline__ void put_atom(Slab<Real>& w, int j, const AtomRec<Real>& a, int64_t gi) {
  w.at[j] = a;
  w.c.x[j] = a.x;
  w.c.y[j] = a.y;
  w.c.z[j] = a.z;
  w.gidx[j] = (int)gi;
}

// Exclusions between a tile of rows (atoms [st, st + c1) of block type bt1,
// one per lane) and atoms [at0, at0 + cnt) of a count-pair partner of type
// bt2: bit k of x set where the smallest separation over the connections
// (ljlk_pose_score.impl.hh:47-67; seps[u * 4 + v]) is below four bonds, of y
// where it is four.  Only partner atoms within four bonds of some connection
// of b1 are compared row by row.
template <typename Real>
__device__ __forceinline__ uint2 partner_masks(const ScoreArgs<Real>& s, int bt1, int nc1, int st, int c1, int bt2,
                                               int nc2, int at0, int cnt, const uint8_t* seps, bool lig, int lane) {
  uint2 m = make_uint2(0u, 0u);
  unsigned bb = 0xffffffffu;  // per connection of b1: the separation from it, a byte each
  bool rel = false;
  if (lane < cnt) {
    const uint32_t cj = load_cpd(s, bt2, nc2, at0 + lane);
    for (int u = 0; u < nc1; ++u) {
      int best = 63;
      for (int v = 0; v < nc2; ++v) best = min(best, (int)seps[u * 4 + v] + (int)((cj >> (8 * v)) & 0xff));
      bb = (bb & ~(0xffu << (8 * u))) | ((unsigned)best << (8 * u));
      rel |= best <= 4;
    }
  }
  const uint32_t c0 = lane < c1 ? load_cpd(s, bt1, nc1, st + lane) : 0x3f3f3f3fu;
  for (unsigned rm = __ballot_sync(0xffffffffu, rel); rm; rm &= rm - 1) {
    const int k = __ffs(rm) - 1;
    const unsigned bk = __shfl_sync(0xffffffffu, bb, k);
    int sep = 5;
    for (int u = 0; u < nc1; ++u) sep = min(sep, (int)((c0 >> (8 * u)) & 0xff) + (int)((bk >> (8 * u)) & 0xff));
    if (lig && (sep == 3 || sep == 4)) sep = 5;
    m.x |= (unsigned)(sep < 4) << k;
    m.y |= (unsigned)(sep == 4) << k;
  }
  return m;
}

// Plan time: the masks of every (block, count-pair partner), one warp each,
// as [word of the partner][atom of the block] from cp_moff on.
template <typename Real>
__global__ void plan_partner_masks_kernel(ScoreArgs<Real> s, uint2* out) {
  const int lane = threadIdx.x & 31;
  const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; row < (int64_t)s.P * s.B;
       row += n_warps) {
    const int4 b1 = s.blk_info[row];
    if (b1.x < 0) continue;
    const int64_t pose0 = row - row % s.B;
    for (int e = 0; e < s.cp_count[row]; ++e) {
      const int64_t k = row * CP_CAP + e;
      const int4 b2 = s.blk_info[pose0 + s.cp_b2[k]];
      const bool lig = (b1.w >> 8) && (b2.w >> 8);
      for (int at0 = 0; at0 < b2.z; at0 += 32)
        for (int st = 0; st < b1.z; st += TILE) {
          const int c1 = min(TILE, b1.z - st);
          const uint2 m = partner_masks(s, b1.x, b1.w & 0xff, st, c1, b2.x, b2.w & 0xff, at0, min(32, b2.z - at0),
                                        s.cp_seps + k * 16, lig, lane);
          if (lane < c1) out[(int64_t)s.cp_moff[k] + (int64_t)(at0 >> 5) * b1.z + st + lane] = m;
        }
    }
  }
}

// The rows: block type, tile start and atoms.
struct RowSide {
  int bt, st, c1;
};

// Stages atoms [at0, at0 + cnt) (cnt <= 32) of a block with exclusions
// against the rows (b1 itself or a count-pair partner) at side-1 atoms
// [base, ...), with the lanes' masks (excluded, weight 0.2) as mask `sp`.
template <typename Real>
__device__ __forceinline__ void stage_masked(const ScoreArgs<Real>& s, Slab<Real>& w, int base, int sp, int64_t off2,
                                             int at0, int cnt, uint2 mask, int lane) {
  const int64_t gi = off2 + at0 + lane;
  if (lane < cnt) put_atom(w, base + lane, s.packed[gi], gi);
  w.smask[sp][lane] = mask;
}

// Keeps, of up to 32 atoms (one per lane), those that can reach b1 (within
// r1 + max_dis of its centre: the cull is exact) and appends them to side 1
// at m; returns how many.
template <typename Real>
__device__ __forceinline__ int stage_culled(Slab<Real>& w, int m, bool valid, const AtomRec<Real>& a, int64_t gi,
                                            Real cx, Real cy, Real cz, Real reach2, int slot, int lane) {
  const Real dx = a.x - cx, dy = a.y - cy, dz = a.z - cz;
  const bool keep = valid && dx * dx + dy * dy + dz * dz < reach2;
  const unsigned km = __ballot_sync(0xffffffffu, keep);
  if (keep) {
    const int j = m + __popc(km & ((1u << lane) - 1u));
    put_atom(w, j, a, gi);
    if (slot >= 0) w.slot[j] = (uint8_t)slot;
  }
  return __popc(km);
}

template <typename Real>
__device__ __forceinline__ EvalCtx<Real> eval_ctx(const ScoreArgs<Real>& s) {
  EvalCtx<Real> c;
  c.lj = s.ljtab;
  c.lk = s.lktab;
  c.far = s.fartab;
  c.elec_k = s.elec_k;
  c.ntp = s.ntp;
  c.max2 = s.g.max_dis * s.g.max_dis;
  c.far2 = s.far_d > Real(0) ? s.far_d * s.far_d : Real(4) * c.max2;
  c.far_dmin = s.g.max_dis - Real(1.5);
  c.far_first = c.far_dmin > Real(4.5) ? c.far_dmin : Real(4.5);
  c.inv_hf = Real(1) / (s.g.max_dis - c.far_dmin);
  c.wt0 = c.wt1 = c.wt2 = c.grid = 0;
  c.g = s.g4;
  c.row0 = 0;
  c.energies = nullptr;
  c.dTdV = nullptr;
  c.stride = 0;
  return c;
}

// The fused kernel.  A work item is (pose p, block b1, candidate range
// [c0, c1) of later blocks b2 >= b1).  Every warp takes items from a global
// ticket, tests b1 against each candidate with the bounding-sphere rule of
// tmol/score/common/sphere_overlap.impl.hh:287-351 (32 per ballot) and
// scores the hits: b1 itself and its count-pair partners with exclusion
// masks, the others as one flat list of atoms (every lane loads one, however
// the blocks' atom counts fall), culled against b1's sphere.  GRAD selects
// the adjoint (which also yields the energies when s.energies is set);
// BLOCK_PAIR selects per-block-pair energies / weights instead of per-pose
// ones: every block then has words of its own.
template <typename Real, bool GRAD, bool BLOCK_PAIR, int TERM, bool COUNT>
__global__ void __launch_bounds__(sizeof(Real) == 4 ? 32 * PAIR_WARPS : 256, 1)
    score_kernel(ScoreArgs<Real> s, int items_per_ticket) {
  if (s.done && *s.done) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Slab<Real>& w = *reinterpret_cast<Slab<Real>*>(smem_raw + warp * slab_bytes<Real>(BLOCK_PAIR && !GRAD));
  const unsigned lemask = 0xffffffffu >> (31 - lane);
  const bool want_E = !GRAD || s.energies != nullptr;
  EvalCtx<Real> ec = eval_ctx(s);
  if (BLOCK_PAIR) {
    ec.energies = s.energies;
    ec.dTdV = s.dTdV;
    ec.stride = (int64_t)s.P * s.B * s.B;
  }
  const int max_words = BLOCK_PAIR ? min(MAXW, s.max_slots) : MAXW;
  long long n_bp = 0, n_ap = 0, n_hp = 0, n_in[2] = {0, 0};

  const int n_work = s.ticket[2];
  for (;;) {
    int t = 0;
    if (lane == 0) t = atomicAdd(s.ticket, 1);
    const int it0 = __shfl_sync(0xffffffffu, t, 0) * items_per_ticket;
    if (it0 >= n_work) break;
    const int it1 = min(it0 + items_per_ticket, n_work);
    for (int item = it0; item < it1; ++item) {
      // item costs for plan_rebalance: measured by the counting instantiation
      const long long t_item = COUNT ? clock64() : 0;
      const int4 wi = s.work[item];
      const int p = wi.x, b1 = wi.y, cand0 = wi.z, cand1 = wi.w;
      const int i1 = p * s.B + b1;
      // what the item starts from, all loaded before the first use: the row's
      // block, sphere and count-pair partners (one per lane, beside their
      // count) and the first 32 candidates
      const int4 bi1 = s.blk_info[i1];
      const Quad<Real> sph1 = reinterpret_cast<const Quad<Real>*>(s.spheres)[i1];
      const int ncp = s.cp_count[i1];
      int cp_b2 = lane < CP_CAP ? s.cp_b2[(int64_t)i1 * CP_CAP + lane] : -1;
      int4 pre_bi = make_int4(-1, 0, 0, 0);
      Quad<Real> pre_s = {0, 0, 0, 0};
      if (cand0 + lane < cand1) {
        pre_bi = s.blk_info[p * s.B + cand0 + lane];
        pre_s = reinterpret_cast<const Quad<Real>*>(s.spheres)[p * s.B + cand0 + lane];
      }
      if (bi1.x < 0) continue;
      if (lane >= ncp) cp_b2 = -1;
      const int n1 = bi1.z;
      RowSide r;
      r.bt = bi1.x;
      if (GRAD && !BLOCK_PAIR) {
        ec.wt0 = s.dTdV[p];
        if (TERM == kTermLJLK) {
          ec.wt1 = s.dTdV[s.P + p];
          ec.wt2 = s.dTdV[2 * s.P + p];
        }
        ec.grid = grid_of_weights<Real, TERM>(ec.wt0, ec.wt1, ec.wt2);
      }
      const Real reach1 = sph1.d + s.g.max_dis;
      const Real reach1_2 = reach1 * reach1 * Real(1.0001);
      E3<Real> acc = {0, 0, 0};
      for (int ti = 0; ti * TILE < n1; ++ti) {
        r.st = ti * TILE;
        r.c1 = min(TILE, n1 - r.st);
        ec.row0 = (int64_t)bi1.y + r.st;
        AtomRec<Real> ra;
        ra.x = ra.y = ra.z = Real(0);
        ra.tf = 0;
        if (lane < r.c1) ra = s.packed[ec.row0 + lane];
        w.row[lane] = ra;
        const unsigned heavy_rows =
            TERM == kTermLJLK ? __ballot_sync(0xffffffffu, lane < r.c1 && (ra.tf & kTfHeavy)) : 0u;
        // what is left to stage: candidate batches, the current batch's
        // blocks with masks (one of them being staged), its other hits
        int next_c = cand0, batch = cand0;
        unsigned spec = 0, hits = 0;
        int sp_n = 0, sp_at = 0, sp_b2 = 0, sp_cp = 0;
        int4 bi2 = make_int4(-1, 0, 0, 0);
        int T = 0, k0 = 0, owned = 0, start = 0;  // pose mode: the flat list of the batch's hits
        bool done = false;
        while (!done) {
          int m = 0, top = M1, nw = 0, nsp = 0;
          for (;;) {
            if (sp_n > 0) {
              // the next word of the block being staged with masks
              const int cnt = min(32, sp_n - sp_at), need = (cnt + 3) & ~3;
              if (nsp == MAXSP || nw >= max_words || m + need > top) break;
              const int src = sp_b2 - batch;
              const int off2 = __shfl_sync(0xffffffffu, bi2.y, src);
              int base = m;
              if (BLOCK_PAIR)
                m += need;
              else
                base = top -= need;
              const int64_t cpe = (int64_t)i1 * CP_CAP + sp_cp;
              // b1 itself: [atom][word] of its block type; a partner: [word][atom]
              uint2 mk = make_uint2(0u, 0u);
              if (lane < r.c1) {
                if (sp_b2 == b1)
                  mk = s.imask[((int64_t)r.bt * s.A + r.st + lane) * s.n_iwords + (sp_at >> 5)];
                else
                  mk = s.pmask[(int64_t)s.cp_moff[cpe] + (int64_t)(sp_at >> 5) * n1 + r.st + lane];
              }
              stage_masked(s, w, base, nsp, (int64_t)off2, sp_at, cnt, mk, lane);
              if (lane == 0) {
                w.desc[nw] = base | (cnt << 8) | ((nsp + 1) << 16);
                w.out[nw] = (int64_t)i1 * s.B + sp_b2;
              }
              if (BLOCK_PAIR && lane < cnt) w.slot[base + lane] = (uint8_t)nw;
              ++nsp;
              ++nw;
              sp_at += 32;
              if (sp_at >= sp_n) sp_n = 0;
            } else if (spec) {
              const int src = __ffs(spec) - 1;
              spec &= spec - 1;
              sp_b2 = batch + src;
              sp_n = __shfl_sync(0xffffffffu, bi2.z, src);
              sp_at = sp_b2 == b1 ? r.st : 0;
              const unsigned pm = __ballot_sync(0xffffffffu, cp_b2 == sp_b2);
              sp_cp = pm ? __ffs(pm) - 1 : 0;
              if (sp_at >= sp_n) sp_n = 0;
            } else if (!BLOCK_PAIR && k0 < T) {
              // as many of the list's atoms as side 1 has room for: all of
              // their loads in flight at once, uncompacted behind m, then
              // culled and moved up in place, 32 at a time
              const int room = min((top - m) & ~31, 32 * (MAXW - nw - ((m + 31) >> 5)));
              if (room <= 0) break;
              const int n = min(room, T - k0);
              for (int q = 0; q < n; q += 32) {
                // bit b of `word` is set where a hit's atoms begin at list
                // position k0 + q + b
                const unsigned pos = (unsigned)(start - k0 - q);
                const unsigned word = __reduce_or_sync(0xffffffffu, pos < 32u ? 1u << pos : 0u);
                const int own = owned + __popc(word & lemask) - 1;
                owned += __popc(word);
                if (q + lane < n) {
                  const int gi = w.hoff[own] + k0 + q + lane;
                  w.gidx[m + q + lane] = gi;
                  copy_async(&w.at[m + q + lane], s.packed + gi);
                }
              }
              copy_wait();
              __syncwarp();
              int src = m;
              for (int q = 0; q < n; q += 32, src += 32) {
                const bool valid = q + lane < n;
                AtomRec<Real> a;
                a.x = a.y = a.z = Real(0);
                a.tf = 0;
                int gi = 0;
                if (valid) {
                  a = w.at[src + lane];
                  gi = w.gidx[src + lane];
                }
                __syncwarp();
                m += stage_culled(w, m, valid, a, gi, sph1.a, sph1.b, sph1.c, reach1_2, -1, lane);
              }
              k0 += n;
              __syncwarp();
            } else if (BLOCK_PAIR && hits) {
              // 32 atoms of the next hit: a word of their own
              if (m + 32 > top || nw >= max_words) break;
              const int src = __ffs(hits) - 1;
              const int off2 = __shfl_sync(0xffffffffu, bi2.y, src), n2 = __shfl_sync(0xffffffffu, bi2.z, src);
              const bool valid = k0 + lane < n2;
              const int64_t gi = (int64_t)off2 + k0 + lane;
              AtomRec<Real> a;
              a.x = a.y = a.z = Real(0);
              a.tf = 0;
              if (valid) a = s.packed[gi];
              const int kept = stage_culled(w, m, valid, a, gi, sph1.a, sph1.b, sph1.c, reach1_2, nw, lane);
              if (kept > 0) {
                if (lane == 0) {
                  w.desc[nw] = m | (kept << 8);
                  w.out[nw] = (int64_t)i1 * s.B + batch + src;
                }
                m += (kept + 3) & ~3;
                ++nw;
              }
              k0 += 32;
              if (k0 >= n2) {
                k0 = 0;
                hits &= hits - 1;
              }
            } else if (next_c < cand1) {
              // the next 32 candidates, loaded while the ones before were
              // processed
              batch = next_c;
              next_c += 32;
              const int b2 = batch + lane;
              bool hit = false;
              bi2 = pre_bi;
              const Quad<Real> s2 = pre_s;
              pre_bi = make_int4(-1, 0, 0, 0);
              {
                // after the last batch: the first again, for the next tile
                const int nx = (next_c < cand1 ? next_c : cand0) + lane;
                if (nx < cand1) {
                  pre_bi = s.blk_info[p * s.B + nx];
                  pre_s = reinterpret_cast<const Quad<Real>*>(s.spheres)[p * s.B + nx];
                }
              }
              if (b2 < cand1) {
                if (bi2.x >= 0) {
                  const Real dx = sub_rn(sph1.a, s2.a), dy = sub_rn(sph1.b, s2.b), dz = sub_rn(sph1.c, s2.c);
                  const Real d2 = add_rn(add_rn(mul_rn(dx, dx), mul_rn(dy, dy)), mul_rn(dz, dz));
                  const Real thr = add_rn(add_rn(sph1.d, s2.d), s.reach);
                  hit = d2 < mul_rn(thr, thr);
                }
                if (s.nbr) s.nbr[(int64_t)i1 * s.B + b2] = hit ? 1 : 0;
              }
              bool masked = b2 == b1;
              for (int k = 0; k < ncp; ++k) masked |= __shfl_sync(0xffffffffu, cp_b2, k) == b2;
              // a screened-out pair is dropped unless it is b1 itself or one
              // of its count-pair partners (bond separation <= 4)
              if (s.skip && hit && !masked &&
                  ((s.skip[(int64_t)i1 * s.skip_words + (b2 >> 5)] >> (b2 & 31)) & 1u))
                hit = false;
              if (COUNT && ti == 0 && hit) {
                const long long n2 = bi2.z;
                n_bp += 1;
                n_ap += b2 == b1 ? n2 * (n2 - 1) / 2 : (long long)n1 * n2;
                if (TERM == kTermLJLK) {
                  const long long h1 = s.bt_n_heavy[r.bt], h2 = s.bt_n_heavy[bi2.x];
                  n_hp += b2 == b1 ? h2 * (h2 - 1) / 2 : h1 * h2;
                }
              }
              spec = __ballot_sync(0xffffffffu, hit && masked);
              hits = __ballot_sync(0xffffffffu, hit && !masked);
              if (!BLOCK_PAIR) {
                // where each hit's atoms begin in the flat list
                const int n = hit && !masked ? bi2.z : 0;
                int inc = n;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                  const int v = __shfl_up_sync(0xffffffffu, inc, o);
                  if (lane >= o) inc += v;
                }
                T = __shfl_sync(0xffffffffu, inc, 31);
                start = n > 0 ? inc - n : 0x7fffffff;
                __syncwarp();
                const unsigned hm = __ballot_sync(0xffffffffu, n > 0);
                if (n > 0) w.hoff[__popc(hm & (lemask >> 1))] = bi2.y - start;
                __syncwarp();
                owned = 0;
              }
              k0 = 0;
            } else {
              done = true;
              break;
            }
          }
          if (!BLOCK_PAIR) {
            // the flat list's words
            const int nf = (m + 31) >> 5;
            if (lane < nf) w.desc[nw + lane] = 32 * lane | (min(32, m - 32 * lane) << 8);
            nw += nf;
          }
          if (nw > 0)
            process_group<Real, GRAD, BLOCK_PAIR, TERM, COUNT>(ec, w, nw, r.c1, ra.x, ra.y, ra.z, heavy_rows, lane,
                                                               acc, n_in);
        }
        __syncwarp();
      }
      if (!BLOCK_PAIR && want_E) {
        const Real v0 = warp_sum(acc.atr);
        const Real v1 = TERM == kTermLJLK ? warp_sum(acc.rep) : Real(0);
        const Real v2 = TERM == kTermLJLK ? warp_sum(acc.lk) : Real(0);
        if (lane == 0) {
          if (v0 != Real(0)) atomicAdd(&s.energies[p], v0);
          if (v1 != Real(0)) atomicAdd(&s.energies[s.P + p], v1);
          if (v2 != Real(0)) atomicAdd(&s.energies[2 * s.P + p], v2);
        }
      }
      if (COUNT && s.item_cost && lane == 0)
        s.item_cost[item] = (int)min((clock64() - t_item) >> 4, (long long)0x7fffffff);
    }
  }
  if (COUNT && s.counts) {
    const long long v[N_COUNTS] = {warp_sum(n_bp), warp_sum(n_ap), warp_sum(n_hp), warp_sum(n_in[0]), warp_sum(n_in[1])};
    if (lane == 0)
      for (int k = 0; k < N_COUNTS; ++k)
        if (v[k]) atomicAdd(&s.counts[k], (unsigned long long)v[k]);
  }
}
