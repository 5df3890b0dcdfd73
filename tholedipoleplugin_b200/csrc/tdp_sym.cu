// tdp_sym.cu -- the all-pairs kernels of the box path (permanent field,
// mutual-field matvec, energy/force/torque), each unordered pair evaluated
// once with both of its sides.
//
// Work decomposition.  Atoms form 32-atom tiles.  The mixed form's kernels take
// warp-sized items (k_field_items, k_energy_items).  In the plain form's, tiles
// form bands and one CTA owns a band pair (p, q), p <= q, and evaluates every
// tile pair (I in band p, J in band q, I <= J).  A warp holds
// the atoms of its I tile(s) in registers (lane = atom) and walks the atoms of
// J along the diagonals of the tile pair, the J-side sums travelling with them
// from lane to lane by shuffles, so that at the end each lane holds the
// J-side sums of "its" J atom.  The FP64 walks pair lane l with J atom
// (l + s) mod 32 at step s.  The mixed form's
// packed walks (f32x2, tdp_f32x2.cuh) pair lane l with J atoms m and m + 16,
// m = (l + s) mod 16, in the two halves of each register; lanes l and l ^ 16
// then hold two copies of the same J sums, added by one xor-16 exchange.
//
// J-side sums of band q.  Plain field kernel: each warp sums into its own area
// of shared memory, the areas are added in warp order at the end.  Plain energy
// kernel: one FP64 area; the warps visit disjoint J tiles within each window
// of band_tiles / 4 steps and a barrier separates the windows, so the order
// of the additions is fixed.
//
// Output.  Plain form: partial sums go to slot s of a [slots][components]
// [n_pad] FP64 buffer -- CTA (p, q) writes the I-side sums of band p into
// slot q and the J-side sums of band q into slot p -- and k_field_slots and
// k_slot_sum add an atom's slots in slot order.  Mixed form: every warp adds its
// sums into one 64-bit fixed-point accumulator (integer addition, independent
// of the order).  Either way results are bitwise deterministic.
//
// Tile pairs are classified as in the reference's arithmetic requires: FOLD
// where the tiles' extents reach half a box (per-pair minimum image with an
// FP64 fallback near the half-box boundary), DAMP where some pair may lie
// within the Thole damping range, MASK (SLOW in the plain energy kernel) on the
// diagonal tile, the ragged last tile and tiles holding covalent partners.
// There self and padding pairs and the partners are left out of the walk; each
// partner pair is evaluated once per side with its M/I scales, by the kernel
// that collects the sums or (plain energy kernel) after the walk.
#include "tdp_frames.cuh"
#include "tdp_f32x2.cuh"
#include "tdp_kernels.cuh"
#include "tdp_pairs.cuh"

#include <cooperative_groups.h>
#include <math.h>

#include <algorithm>

namespace cg = cooperative_groups;

namespace tdp {

namespace {

constexpr int kSymWarps = 4;
constexpr int kSymThreads = 32 * kSymWarps;
constexpr unsigned kFull = 0xffffffffu;

// Band pair of CTA k, enumerated q = 0, 1, ... and p = 0..q: k = q(q+1)/2 + p.
__device__ __forceinline__ void band_pair(int k, int& p, int& q) {
    int qq = (int)((sqrt(8.0 * (double)k + 1.0) - 1.0) * 0.5);
    while ((qq + 1) * (qq + 2) / 2 <= k) qq++;
    while (qq * (qq + 1) / 2 > k) qq--;
    q = qq;
    p = k - qq * (qq + 1) / 2;
}

// FP32 walks end the damping where the exponent x = a u^3 is 25, half of what
// P.damp_r2 stands for: the largest departure of a factor from 1 there is
// (1 + x + 1.5 x^2) exp(-x) = 1.4e-8, under half an ulp of 1 (3.0e-8), so every
// FP32 factor beyond is 1 either way, and fewer tile pairs take the damped
// walk (its range is 0.58 instead of 0.73 nm for water).
constexpr float kDampRange32 = 0.62996f;   // (25/50)^(2/3)

// Geometry of a tile pair: displacement of J's centre from I's (FP64, minimum
// image), whether any pair needs per-pair folding, whether any pair can be
// within the damping range.
struct TileGeom {
    double dcx, dcy, dcz;
    bool fold;
    bool near;
    unsigned fmask;   // dimensions in which some pair may need folding (bit k: dimension k)
};

__device__ __forceinline__ TileGeom tile_geom(const PairParams& P, double damp_r2, double4 cA, double4 eA, double4 cB,
                                              double4 eB) {
    TileGeom g;
    g.dcx = cB.x - cA.x;
    g.dcy = cB.y - cA.y;
    g.dcz = cB.z - cA.z;
    g.fold = false;
    g.fmask = 0u;
    if (P.periodic) {
        g.dcx = fold_d(g.dcx, P.box[0], P.inv_box[0]);
        g.dcy = fold_d(g.dcy, P.box[1], P.inv_box[1]);
        g.dcz = fold_d(g.dcz, P.box[2], P.inv_box[2]);
        g.fmask = (fabs(g.dcx) + eA.x + eB.x >= P.half_box_tol[0] ? 1u : 0u) |
                  (fabs(g.dcy) + eA.y + eB.y >= P.half_box_tol[1] ? 2u : 0u) |
                  (fabs(g.dcz) + eA.z + eB.z >= P.half_box_tol[2] ? 4u : 0u);
        g.fold = fabs(g.dcx) + eA.x + eB.x >= P.half_box_tol[0] || fabs(g.dcy) + eA.y + eB.y >= P.half_box_tol[1] ||
                 fabs(g.dcz) + eA.z + eB.z >= P.half_box_tol[2];
    }
    // Smallest minimum-image distance any pair of the two tiles can have: per
    // dimension the periodic distance is a metric, so it is at least the
    // centres' folded distance minus both extents.
    double gx = fmax(fabs(g.dcx) - eA.x - eB.x, 0.0);
    double gy = fmax(fabs(g.dcy) - eA.y - eB.y, 0.0);
    double gz = fmax(fabs(g.dcz) - eA.z - eB.z, 0.0);
    g.near = gx * gx + gy * gy + gz * gz < damp_r2;
    return g;
}

// Exact FP64 minimum-image displacement p_j - p_i (the reference's own
// arithmetic), for FP32 pairs near the half-box.
__device__ __forceinline__ d3 exact_delta(const PairParams& P, const double* __restrict__ pos, int i, int j) {
    d3 d = ld3(pos + 3 * j) - ld3(pos + 3 * i);
    if (P.periodic) {
        d.x = fold_d(d.x, P.box[0], P.inv_box[0]);
        d.y = fold_d(d.y, P.box[1], P.inv_box[1]);
        d.z = fold_d(d.z, P.box[2], P.inv_box[2]);
    }
    return d;
}

// p_j - p_i from j's position and i's shifted into j's image; fold: bits of the
// dimensions that need folding.
template <bool FOLD>
__device__ __forceinline__ void pair_delta(const PairParams& P, unsigned fold, double pjx, double pjy, double pjz,
                                           double oix, double oiy, double oiz, double& dx, double& dy, double& dz) {
    dx = pjx - oix;
    dy = pjy - oiy;
    dz = pjz - oiz;
    if (FOLD) {
        if (fold & 1u) dx = fold_magic(dx, P.box[0], P.inv_box[0], __double2hiint(P.half_box_tol[0]));
        if (fold & 2u) dy = fold_magic(dy, P.box[1], P.inv_box[1], __double2hiint(P.half_box_tol[1]));
        if (fold & 4u) dz = fold_magic(dz, P.box[2], P.inv_box[2], __double2hiint(P.half_box_tol[2]));
    }
}

// The position of an I-tile atom shifted by the whole-box image that the tile
// pair chose.
__device__ __forceinline__ void shift_into(const TileGeom& g, double4 cA, double4 cB, double px, double py, double pz,
                                           double& ox, double& oy, double& oz) {
    ox = px + ((cB.x - cA.x) - g.dcx);
    oy = py + ((cB.y - cA.y) - g.dcy);
    oz = pz + ((cB.z - cA.z) - g.dcz);
}

// Pairs of the diagonal walk that are left out: self, padding, listed
// partners, and on the diagonal tile the second visit of every pair (steps
// 17..31 and the upper half of step 16 repeat steps 15..1 and 16).
__device__ __forceinline__ bool skip_pair(int s, int lane, int i, int j, int n, unsigned partners, int jj, bool diag) {
    bool skip = i >= n || j >= n || ((partners >> jj) & 1u);
    if (diag) skip = skip || s == 0 || s > 16 || (s == 16 && lane >= 16);
    return skip;
}

// Bits of the J-tile atoms listed as covalent partners of atom i.
__device__ __forceinline__ unsigned partner_bits(const int* __restrict__ exc_j, int e0, int e1, int jbase) {
    unsigned b = 0u;
    for (int e = e0; e < e1; e++) {
        unsigned off = (unsigned)(exc_j[e] - jbase);
        if (off < 32u) b |= 1u << off;
    }
    return b;
}

template <class R>
__device__ __forceinline__ void store_operand(typename Vec4T<R>::type* v, int k, d3 a, double t) {
    typename Vec4T<R>::type o;
    o.x = (R)a.x;
    o.y = (R)a.y;
    o.z = (R)a.z;
    o.w = (R)t;
    v[k] = o;
}

// 64-bit fixed-point accumulator of the mixed form (Dev::fixacc).
struct FixAcc {
    unsigned long long* acc;
    int* err;
    double scale, limit;
};

// Adds v to the accumulator word; a sum at or beyond the limit (or not finite)
// flags the error instead of wrapping.
__device__ __forceinline__ void fix_add(const FixAcc& F, size_t k, double v) {
    if (v == 0.0) return;
    if (!(fabs(v) < F.limit)) {
        atomicExch(F.err, 1);
        return;
    }
    atomicAdd(F.acc + k, (unsigned long long)__double2ll_rn(v * F.scale));
}

// ---------------------------------------------------------------------------
// Field kernels: KIND 0 = permanent field (records: posq + lab dipole/thole),
// KIND 1 = mutual-field matvec T*v (records: posq + v/thole).
// ---------------------------------------------------------------------------
// The plain form's J records, one 16-byte piece of every atom after the other:
// a warp reads 32 consecutive pieces without bank conflicts (8 wavefronts for
// a 32-byte record of each lane, against 16 when the records lie whole).

struct Rec64 {
    double2 *xy, *zx, *yz, *qt;   // (x, y), (z, vx), (vy, vz), (q, t)
    double* c;                    // 1 / t^3
};

// Two I atoms of a lane against the J tile at j0: both sides of every pair.
// MASK: bit jj of m[k] is the pair (slot k, J atom jj); the other walks take all.
template <int KIND, bool FOLD, bool DAMP, bool MASK>
__device__ __forceinline__ void field_walk64(const PairParams& P, const Rec64& T, int lane, int j0,
                                             const double (&o)[2][3], const double (&v)[2][3], const double (&q)[2],
                                             const double (&ti)[2], const double (&c3)[2], const unsigned (&m)[2],
                                             unsigned fold, int s0, int s1, double (&f)[2][3], double (&g)[3]) {
    const int nxt = (lane + 1) & 31;
#pragma unroll 1
    for (int s = s0; s < s1; s++) {
        const int jj = (lane + s) & 31;
        const double2 xy = T.xy[j0 + jj], zx = T.zx[j0 + jj], yz = T.yz[j0 + jj];
        double2 qt = make_double2(0.0, 0.0);
        if (KIND == 0 || DAMP) qt = T.qt[j0 + jj];
        const double wx = zx.y, wy = yz.x, wz = yz.y;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            double dx, dy, dz;
            pair_delta<FOLD>(P, fold, xy.x, xy.y, zx.x, o[k][0], o[k][1], o[k][2], dx, dy, dz);
            const double r2 = dx * dx + dy * dy + dz * dz;
            double rinv = rsqrt_step(r2);
            if (MASK) rinv = (m[k] >> jj) & 1u ? rinv : 0.0;
            const double rinv2 = rinv * rinv;
            double rr3 = rinv * rinv2;
            double rr5 = 3.0 * rr3 * rinv2;
            if (DAMP && r2 < (double)P.damp_r2 && ti[k] * qt.y != 0.0) {
                // x = min(t_i, t_j) (r / (t_i t_j))^3
                const double x = fmin(ti[k], qt.y) * (r2 * r2 * rinv) * (c3[k] * T.c[j0 + jj]);
                if (x < 50.0) {
                    const double ex = exp(-x);
                    rr3 *= 1.0 - ex;
                    rr5 *= 1.0 - (1.0 + x) * ex;
                }
            }
            double a = rr5 * (wx * dx + wy * dy + wz * dz);
            double b = rr5 * (v[k][0] * dx + v[k][1] * dy + v[k][2] * dz);
            if (KIND == 0) {
                a = fma(-rr3, qt.x, a);
                b = fma(rr3, q[k], b);
            }
            f[k][0] = fma(a, dx, fma(-rr3, wx, f[k][0]));
            f[k][1] = fma(a, dy, fma(-rr3, wy, f[k][1]));
            f[k][2] = fma(a, dz, fma(-rr3, wz, f[k][2]));
            g[0] = fma(b, dx, fma(-rr3, v[k][0], g[0]));
            g[1] = fma(b, dy, fma(-rr3, v[k][1], g[1]));
            g[2] = fma(b, dz, fma(-rr3, v[k][2], g[2]));
        }
        g[0] = __shfl_sync(kFull, g[0], nxt);
        g[1] = __shfl_sync(kFull, g[1], nxt);
        g[2] = __shfl_sync(kFull, g[2], nxt);
    }
}

// ---------------------------------------------------------------------------
// Packed FP32 walk over J-atom pairs: the halves of every 64-bit register are
// J atoms m and m + 16 of the tile (records pair-interleaved in a per-warp
// shared tile), so the I-side operands are loop-invariant broadcasts and the
// J-side sums stay packed.  Lane l takes pair m = (l + s) & 15 at step s and
// passes its packed J-side sums one lane on; lanes l and l ^ 16 hold two
// partial copies of the same pair, added by one xor-16 exchange at the end.
// Each lane carries NS I atoms; both sides of every pair are evaluated
// (calculateInducedDipolePairIxn and calculateFixedDipoleFieldPairIxn,
// RTDF.cpp:766-818 and :678-713).
// ---------------------------------------------------------------------------
struct FPackedTile {
    float4 p0[16], p1[16];   // (x, x', y, y'), (z, z', q, q')   (' = atom m + 16)
    float4 v0[16], v1[16];   // (vx, vx', vy, vy'), (vz, vz', t, t')
};

__device__ __forceinline__ void stage_fpacked(FPackedTile& T, int lane, float4 p, float4 v) {
    const int m = lane & 15, h = lane >> 4;
    float* p0 = reinterpret_cast<float*>(&T.p0[m]);
    float* p1 = reinterpret_cast<float*>(&T.p1[m]);
    float* v0 = reinterpret_cast<float*>(&T.v0[m]);
    float* v1 = reinterpret_cast<float*>(&T.v1[m]);
    p0[h] = p.x;
    p0[2 + h] = p.y;
    p1[h] = p.z;
    p1[2 + h] = p.w;
    v0[h] = v.x;
    v0[2 + h] = v.y;
    v1[h] = v.z;
    v1[2 + h] = v.w;
}

// Loop-invariant operands of one I atom.
struct XSlot {
    f2 OX, OY, OZ, VX, VY, VZ, NQ;   // NQ = -q
    float t;
    int i;
};

__device__ __forceinline__ XSlot xslot(int i, float ox, float oy, float oz, float q, float4 v) {
    XSlot x;
    x.OX = bc2(ox);
    x.OY = bc2(oy);
    x.OZ = bc2(oz);
    x.VX = bc2(v.x);
    x.VY = bc2(v.y);
    x.VZ = bc2(v.z);
    x.NQ = bc2(-q);
    x.t = v.w;
    x.i = i;
    return x;
}

// One I atom against J atoms (m, m + 16): I-side sums into F*, J-side into G*,
// both with the opposite sign of the field (the walk's caller flips them), so
// that every term is a plain product-sum with -rr5.
// MASK: bit m of mk (bit m + 16 for the second half) says whether the pair counts.
template <int KIND, bool FOLD, bool DAMP, bool MASK = false>
__device__ __forceinline__ void xslot_pairs(const PairParams& P, const double* __restrict__ pos, const XSlot& x,
                                            unsigned mk, int m, int ja, f2 PX, f2 PY, f2 PZ, f2 QJ, f2 VJX, f2 VJY,
                                            f2 VJZ, float tja, float tjb, unsigned fm, f2 Lx, f2 Ly, f2 Lz, f2 Ix,
                                            f2 Iy, f2 Iz,
                                            f2 NTx, f2 NTy, f2 NTz, float damp_r2, f2& FX, f2& FY, f2& FZ,
                                            f2& GX, f2& GY, f2& GZ) {
    f2 DX = sub2(PX, x.OX), DY = sub2(PY, x.OY), DZ = sub2(PZ, x.OZ);
    if (FOLD) {
        // Fold the dimensions of fm.  Q = d^2 - t^2 (t = half a box minus 16
        // ulp) is negative unless the pair lies within the margin of half a
        // box; AND-ing the Q words keeps sign bits 31 (low half) and 63 (high
        // half) set only if every Q of that half is negative.
        f2 neg = ~0ull;
        if (fm & 1u) {
            DX = fold2(DX, Lx, Ix);
            neg &= fma2(DX, DX, NTx);
        }
        if (fm & 2u) {
            DY = fold2(DY, Ly, Iy);
            neg &= fma2(DY, DY, NTy);
        }
        if (fm & 4u) {
            DZ = fold2(DZ, Lz, Iz);
            neg &= fma2(DZ, DZ, NTz);
        }
        const f2 flag = ~neg & 0x8000000080000000ull;
        if (flag) {
            const bool amb_a = (flag >> 31) & 1ull, amb_b = (flag >> 63) != 0ull;
            float ax, bx, ay, by, az, bz;
            un2(DX, ax, bx);
            un2(DY, ay, by);
            un2(DZ, az, bz);
            // Within 16 ulp of half a box: the reference's FP64 minimum image.
            if (amb_a && x.i < P.n && ja < P.n) {
                d3 e = exact_delta(P, pos, x.i, ja);
                ax = (float)e.x;
                ay = (float)e.y;
                az = (float)e.z;
            }
            if (amb_b && x.i < P.n && ja + 16 < P.n) {
                d3 e = exact_delta(P, pos, x.i, ja + 16);
                bx = (float)e.x;
                by = (float)e.y;
                bz = (float)e.z;
            }
            DX = pk2(ax, bx);
            DY = pk2(ay, by);
            DZ = pk2(az, bz);
        }
    }
    const f2 R2 = fma2(DX, DX, fma2(DY, DY, mul2(DZ, DZ)));
    float r2a, r2b;
    un2(R2, r2a, r2b);
    if (MASK) {
        // A pair that does not count gets an infinite distance: every term is 0.
        r2a = (mk >> m) & 1u ? r2a : INFINITY;
        r2b = (mk >> (m + 16)) & 1u ? r2b : INFINITY;
    }
    const f2 RINV = pk2(rsqrt_r(r2a), rsqrt_r(r2b));
    const f2 RINV2 = mul2(RINV, RINV);
    f2 RR3 = mul2(RINV, RINV2);
    f2 NRR5 = mul2(RR3, mul2(RINV2, bc2(-3.0f)));   // -rr5
    if (DAMP) {
        if (r2a < damp_r2 || r2b < damp_r2) {
            float ra, rb, r3a, r3b, r5a, r5b;
            un2(RINV, ra, rb);
            un2(RR3, r3a, r3b);
            un2(NRR5, r5a, r5b);
            r5a = -r5a;
            r5b = -r5b;
            damp_field<float>(r2a, ra, x.t, tja, damp_r2, r3a, r5a);
            damp_field<float>(r2b, rb, x.t, tjb, damp_r2, r3b, r5b);
            RR3 = pk2(r3a, r3b);
            NRR5 = pk2(-r5a, -r5b);
        }
    }
    if (KIND == 1) {
        // Mutual field, both sums negated: -f_i += rr3 v_j - (rr5 v_j.d) d,
        // -f_j += rr3 v_i - (rr5 v_i.d) d.
        const f2 DDJ = mul2(NRR5, fma2(VJX, DX, fma2(VJY, DY, mul2(VJZ, DZ))));
        const f2 DDI = mul2(NRR5, fma2(x.VX, DX, fma2(x.VY, DY, mul2(x.VZ, DZ))));
        FX = fma2(RR3, VJX, fma2(DDJ, DX, FX));
        FY = fma2(RR3, VJY, fma2(DDJ, DY, FY));
        FZ = fma2(RR3, VJZ, fma2(DDJ, DZ, FZ));
        GX = fma2(RR3, x.VX, fma2(DDI, DX, GX));
        GY = fma2(RR3, x.VY, fma2(DDI, DY, GY));
        GZ = fma2(RR3, x.VZ, fma2(DDI, DZ, GZ));
    } else {
        // Permanent field: a = rr3 q_j - rr5 m_j.d, b = rr3 q_i + rr5 m_i.d;
        // -f_i += d a + m_j rr3;  -f_j += m_i rr3 - d b, with nb = -b.
        const f2 A = fma2(NRR5, fma2(VJX, DX, fma2(VJY, DY, mul2(VJZ, DZ))), mul2(RR3, QJ));
        const f2 NB = fma2(NRR5, fma2(x.VX, DX, fma2(x.VY, DY, mul2(x.VZ, DZ))), mul2(RR3, x.NQ));
        FX = fma2(VJX, RR3, fma2(DX, A, FX));
        FY = fma2(VJY, RR3, fma2(DY, A, FY));
        FZ = fma2(VJZ, RR3, fma2(DZ, A, FZ));
        GX = fma2(x.VX, RR3, fma2(DX, NB, GX));
        GY = fma2(x.VY, RR3, fma2(DY, NB, GY));
        GZ = fma2(x.VZ, RR3, fma2(DZ, NB, GZ));
    }
}

// Steps [s0, s1) of the walk of NS I tiles (lane = atom of each) over one J
// tile.  g: the J-side sums of atom ((lane + s1) & 15) | (lane & 16).
template <int KIND, int NS, bool FOLD, bool DAMP, bool MASK>
__device__ __forceinline__ void field_walk_ns(const PairParams& P, const double* __restrict__ pos,
                                              const FPackedTile& T, int lane, int jbase, const XSlot (&x)[NS],
                                              const unsigned (&mk)[NS], const unsigned (&fm)[NS], float damp_r2,
                                              int s0, int s1,
                                              float (&f)[NS][3], float (&g)[3]) {
    const int nxt = (lane + 1) & 31;
    f2 Lx = 0, Ly = 0, Lz = 0, Ix = 0, Iy = 0, Iz = 0, NTx = 0, NTy = 0, NTz = 0;
    if (FOLD) {
        Lx = bc2(-(float)P.box[0]);
        Ly = bc2(-(float)P.box[1]);
        Lz = bc2(-(float)P.box[2]);
        Ix = bc2((float)P.inv_box[0]);
        Iy = bc2((float)P.inv_box[1]);
        Iz = bc2((float)P.inv_box[2]);
        NTx = bc2(-(float)(P.half_box_tol[0] * P.half_box_tol[0]));
        NTy = bc2(-(float)(P.half_box_tol[1] * P.half_box_tol[1]));
        NTz = bc2(-(float)(P.half_box_tol[2] * P.half_box_tol[2]));
    }
    f2 F[NS][3];               // I side, packed over (m, m + 16)
#pragma unroll
    for (int k = 0; k < NS; k++) F[k][0] = F[k][1] = F[k][2] = 0;
    f2 GX = 0, GY = 0, GZ = 0;   // J side (packed atoms m, m + 16)
    // One step is already 2 NS independent pairs: no unrolling (the walk's
    // variants must stay small enough for the instruction cache).
#pragma unroll 1
    for (int s = s0; s < s1; s++) {
        const int m = (lane + s) & 15;
        const float4 a = T.p0[m], b = T.p1[m], c = T.v0[m], d = T.v1[m];
        const f2 PX = pk2(a.x, a.y), PY = pk2(a.z, a.w), PZ = pk2(b.x, b.y), QJ = pk2(b.z, b.w);
        const f2 VJX = pk2(c.x, c.y), VJY = pk2(c.z, c.w), VJZ = pk2(d.x, d.y);
#pragma unroll
        for (int k = 0; k < NS; k++)
            xslot_pairs<KIND, FOLD, DAMP, MASK>(P, pos, x[k], mk[k], m, jbase + m, PX, PY, PZ, QJ, VJX, VJY, VJZ, d.z,
                                                d.w, fm[k], Lx, Ly, Lz, Ix, Iy, Iz, NTx, NTy, NTz, damp_r2, F[k][0],
                                                F[k][1], F[k][2], GX, GY, GZ);
        GX = __shfl_sync(kFull, GX, nxt);
        GY = __shfl_sync(kFull, GY, nxt);
        GZ = __shfl_sync(kFull, GZ, nxt);
    }
    // F and G hold the negated sums (xslot_pairs).
    float lo, hi;
#pragma unroll
    for (int k = 0; k < NS; k++)
#pragma unroll
        for (int c = 0; c < 3; c++) {
            un2(F[k][c], lo, hi);
            f[k][c] = -(lo + hi);
        }
    // Lanes l and l ^ 16 hold the two copies of atoms (m, m + 16), m = (l + s1) & 15.
    const f2 Js[3] = {GX, GY, GZ};
#pragma unroll
    for (int c = 0; c < 3; c++) {
        un2(Js[c], lo, hi);
        const float olo = __shfl_xor_sync(kFull, lo, 16), ohi = __shfl_xor_sync(kFull, hi, 16);
        g[c] = -(lane < 16 ? lo + olo : hi + ohi);
    }
}

// A float sum into the accumulator: v 2^k is exact, so the only rounding is
// that of the accumulator's unit.
__device__ __forceinline__ void fix_add(const FixAcc& F, size_t k, float v) {
    if (v == 0.0f) return;
    if (!(fabsf(v) < (float)F.limit)) {
        atomicExch(F.err, 1);
        return;
    }
    atomicAdd(F.acc + k, (unsigned long long)__float2ll_rn(v * (float)F.scale));
}

// Mixed-form field kernel: KIND 0 = permanent field (operand: lab dipoles, or
// m + mu0 in the fused start), KIND 1 = mutual-field matvec.  One warp is one
// item: NS I tiles in registers against J tiles [c L, c L + L), and of each
// walk the steps of its part (gridDim.y parts).  Items are independent: the J
// records come from L2 into the warp's own packed tile, the J-side sums of a
// tile pair go straight into the fixed-point accumulator, so no block waits at
// a barrier and any number of tiles splits evenly.  Pairs that do not count
// (self, padding, the second visit on a diagonal tile, partners whose scale is
// not 1) are masked out; k_field_done adds the scaled partners.
//
// Bound by the FP32 pipe and issue (61 FMA-pipe instructions of about 90 a
// step of four pairs).  The kernel before it owned a band pair per 4-warp
// block, summed the J side in shared memory and flushed 2 x 3 x 512 sums; its
// bands had to shrink with the system, which left warps with one I tile (half
// the work per J load and shuffle) or none.  Matvec, before -> now: 19.7 ->
// 12 us at 648 atoms (with k_field_done), 94 -> 41 at 3,993, 242 -> 169 at
// 12,288, 8730 -> 6890 at 98,304 (in Hilbert order, undamped beyond exponent
// 25; 43, 175 and 6950 before these).  NS = 4 is slower (7126 us there, 321 at
// 12,288): the tiles of an item share the fold and damping variant of a walk.
template <int KIND, int NS>
__global__ void __launch_bounds__(32, 16) k_field_items(
    PairParams P, int L, const float4* __restrict__ posq, const float4* __restrict__ jvec,
    const double4* __restrict__ tctr, const double4* __restrict__ text, const double* __restrict__ pos,
    const int* __restrict__ exc_off, const int* __restrict__ exc_j, const double* __restrict__ exc_scale,
    const int2* __restrict__ exc_tiles, int n_pad, FixAcc fix, CgStop stop) {
    if (stop.stopped()) return;
    __shared__ FPackedTile T;
    __shared__ double s_my[3 * NS][32];   // I-side sums
    const int lane = threadIdx.x;
    // Item -> (I group a, J chunk c): square blocks of B = max(L, NS) tiles, p <= q.
    int p, q, a, c;
    if (L >= NS) {
        const int r = L / NS;
        band_pair(blockIdx.x / r, p, q);
        a = p * r + blockIdx.x % r;
        c = q;
    } else {
        const int r = NS / L;
        band_pair(blockIdx.x / r, p, q);
        a = p;
        c = q * r + blockIdx.x % r;
    }
    const int I0 = a * NS, J0 = c * L, J1 = min(J0 + L, P.n_tiles);
    if (I0 >= P.n_tiles || J1 <= max(J0, I0)) return;
    const int s0 = 16 * blockIdx.y / gridDim.y, s1 = 16 * (blockIdx.y + 1) / gridDim.y;
    const float damp_r2 = kDampRange32 * P.damp_r2;

    float4 pi[NS], vi[NS];
    int2 et[NS];
    int e0[NS], e1[NS];
    unsigned own[NS];
#pragma unroll
    for (int k = 0; k < NS; k++) {
        const int I = I0 + k, i = I * 32 + lane;
        pi[k] = vi[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        et[k] = make_int2(1 << 30, -1);
        e0[k] = e1[k] = 0;
        own[k] = 0u;
        if (I < P.n_tiles) {
            pi[k] = posq[i];
            vi[k] = jvec[i];
            et[k] = exc_tiles[I];
            if (i < P.n) {
                own[k] = ~0u;
                e0[k] = exc_off[i];
                e1[k] = exc_off[i + 1];
            }
        }
    }
    // The item's NS x L tile-pair geometries (FP64), one per lane, read by shuffles.
    float gdx = 0.f, gdy = 0.f, gdz = 0.f;
    unsigned gfl = 0u;
    {
        const int k = lane / L, I = I0 + k, J = J0 + lane % L;
        if (k < NS && I < P.n_tiles && J < P.n_tiles) {
            const TileGeom g = tile_geom(P, (double)damp_r2, tctr[I], text[I], tctr[J], text[J]);
            gdx = (float)g.dcx;
            gdy = (float)g.dcy;
            gdz = (float)g.dcz;
            gfl = g.fmask | (g.fold ? 8u : 0u) | (g.near ? 16u : 0u);
        }
    }
#pragma unroll
    for (int k = 0; k < 3 * NS; k++) s_my[k][lane] = 0.0;
    int J = max(J0, I0);
    float4 pj = posq[J * 32 + lane], vj = jvec[J * 32 + lane];
    for (; J < J1; J++) {
        __syncwarp();
        stage_fpacked(T, lane, pj, vj);
        __syncwarp();
        if (J + 1 < J1) {   // the next tile's records arrive during the walk
            pj = posq[(J + 1) * 32 + lane];
            vj = jvec[(J + 1) * 32 + lane];
        }
        const int jbase = J * 32;
        XSlot x[NS];
        unsigned mk[NS], fm[NS], fl = 0u;
        bool masked = false;
        const unsigned real = J == P.n_tiles - 1 && (P.n & 31) ? (1u << (P.n & 31)) - 1u : ~0u;
#pragma unroll
        for (int k = 0; k < NS; k++) {
            const int I = I0 + k, src = k * L + (J - J0);
            const float dx = __shfl_sync(kFull, gdx, src), dy = __shfl_sync(kFull, gdy, src),
                        dz = __shfl_sync(kFull, gdz, src);
            const unsigned fk = __shfl_sync(kFull, gfl, src);
            mk[k] = own[k] & real;
            if (I > J) mk[k] = 0u;
            if (I == J) mk[k] &= ~((2u << lane) - 1u);   // each pair of a diagonal tile once: j > i
            if (J >= et[k].x && J <= et[k].y)
                for (int e = e0[k]; e < e1[k]; e++) {
                    const unsigned off = (unsigned)(exc_j[e] - jbase);
                    if (off < 32u && exc_scale[e] != 1.0) mk[k] &= ~(1u << off);
                }
            masked = masked || mk[k] != ~0u;
            fl |= fk;
            fm[k] = fk & 7u;
            x[k] = xslot(I * 32 + lane, pi[k].x - dx, pi[k].y - dy, pi[k].z - dz, pi[k].w, vi[k]);
        }
        float f[NS][3], g[3];
        if (__any_sync(kFull, masked))
            field_walk_ns<KIND, NS, true, true, true>(P, pos, T, lane, jbase, x, mk, fm, damp_r2, s0, s1, f, g);
        else if (fl & 8u) {
            if (fl & 16u)
                field_walk_ns<KIND, NS, true, true, false>(P, pos, T, lane, jbase, x, mk, fm, damp_r2, s0, s1, f, g);
            else
                field_walk_ns<KIND, NS, true, false, false>(P, pos, T, lane, jbase, x, mk, fm, damp_r2, s0, s1, f, g);
        } else if (fl & 16u) {
            field_walk_ns<KIND, NS, false, true, false>(P, pos, T, lane, jbase, x, mk, fm, damp_r2, s0, s1, f, g);
        } else {
            field_walk_ns<KIND, NS, false, false, false>(P, pos, T, lane, jbase, x, mk, fm, damp_r2, s0, s1, f, g);
        }
        const int jl = ((lane + s1) & 15) | (lane & 16);
#pragma unroll
        for (int k = 0; k < 3; k++) fix_add(fix, (size_t)k * n_pad + jbase + jl, g[k]);
#pragma unroll
        for (int k = 0; k < NS; k++)
#pragma unroll
            for (int d = 0; d < 3; d++) s_my[3 * k + d][lane] += (double)f[k][d];
    }
#pragma unroll
    for (int k = 0; k < NS; k++)
#pragma unroll
        for (int d = 0; d < 3; d++) fix_add(fix, (size_t)d * n_pad + (I0 + k) * 32 + lane, s_my[3 * k + d][lane]);
}

// Atom k's covalent partner e, which the walks masked out, one-sided with its
// scale (FP64 displacement and arithmetic on the pair records).  KIND 0: M
// scale; 1: I scale; fused (KIND 0, operand P = m + mu0): M field(q, P) +
// (I - M) T mu0 with mu0 = P - m, the second term also where M = 1.
template <int KIND, class V4>
__device__ __forceinline__ void add_partner(const PairParams& P, int fused, const V4* __restrict__ posq,
                                            const V4* __restrict__ jvec, const V4* __restrict__ lab,
                                            const double* __restrict__ pos, const int* __restrict__ exc_j,
                                            const double* __restrict__ exc_m, const double* __restrict__ exc_s, int k,
                                            int e, double ti, double (&f)[3]) {
    const double sc = KIND == 0 ? exc_m[e] : exc_s[e], ds = fused ? exc_s[e] - sc : 0.0;
    if ((sc == 0.0 || sc == 1.0) && ds == 0.0) return;
    const int j = exc_j[e];
    const d3 d = exact_delta(P, pos, k, j);
    const double r2 = dot(d, d);
    const V4 vj = jvec[j];
    double t[3] = {0.0, 0.0, 0.0};
    if (KIND == 0)
        pair_fixed<double, true>(d.x, d.y, d.z, r2, (double)posq[j].w, (double)vj.x, (double)vj.y, (double)vj.z, ti,
                                 (double)vj.w, (double)P.damp_r2, t[0], t[1], t[2]);
    else
        pair_matvec<double, true>(d.x, d.y, d.z, r2, (double)vj.x, (double)vj.y, (double)vj.z, ti, (double)vj.w,
                                  (double)P.damp_r2, t[0], t[1], t[2]);
    if (sc != 1.0)
        for (int c = 0; c < 3; c++) f[c] += sc * t[c];
    if (ds != 0.0) {
        const V4 mj = lab[j];
        double u[3] = {0.0, 0.0, 0.0};
        pair_matvec<double, true>(d.x, d.y, d.z, r2, (double)vj.x - (double)mj.x, (double)vj.y - (double)mj.y,
                                  (double)vj.z - (double)mj.z, ti, (double)vj.w, (double)P.damp_r2, u[0], u[1], u[2]);
        for (int c = 0; c < 3; c++) f[c] += ds * u[c];
    }
}

// Fixed-point sums -> partial slot 0, clearing them, plus the partner pairs.
template <int KIND>
__global__ void k_field_done(PairParams P, int fused, const float4* __restrict__ posq, const float4* __restrict__ jvec,
                             const float4* __restrict__ lab, const double* __restrict__ pos,
                             const int* __restrict__ exc_off, const int* __restrict__ exc_j,
                             const double* __restrict__ exc_m, const double* __restrict__ exc_s, int n_pad,
                             unsigned long long* __restrict__ acc, double inv_scale, double* __restrict__ out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n_pad) return;
    double f[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        f[c] = (double)(long long)acc[(size_t)c * n_pad + k] * inv_scale;
        acc[(size_t)c * n_pad + k] = 0ull;
    }
    if (k < P.n) {
        const double ti = (double)jvec[k].w;
        for (int e = exc_off[k]; e < exc_off[k + 1]; e++)
            add_partner<KIND>(P, fused, posq, jvec, lab, pos, exc_j, exc_m, exc_s, k, e, ti, f);
    }
#pragma unroll
    for (int c = 0; c < 3; c++) out[(size_t)c * n_pad + k] = f[c];
}

// Plain form: one CTA per band pair and part of the walks, BT / 2 warps with
// two I tiles each (see the top of the file).  Sums into slots of `partial`, part
// y's from slot y * bands on.
//
// Bound by the latency of the FP64 chain: 37 FP64 operations a pair (43 with
// the damped and masked tiles) keep the FP64 pipe 55 % busy with 16 warps an SM.
// Hence two independent pairs a step, no unrolling (unrolled twice, the five
// walks no longer share the instruction cache: 452 instead of 385 us), and
// everything a walk does not need reread per J tile to stay at 122 registers.
// The kernel before (one I tile a warp in narrow bands, whole 32-byte records,
// library 1/sqrt and floor) against this one, matvec: 47 -> 30 us at 1,029
// atoms, 227 -> 83 at 3,993, 516 -> 372 at 12,288, 2265 -> 2031 at 31,944.
template <int KIND>
__global__ void __launch_bounds__(128, 4)
    k_field_bands(PairParams P, int BT, const double4* __restrict__ posq, const double4* __restrict__ jvec,
                  const double4* __restrict__ tctr, const double4* __restrict__ text, const int* __restrict__ exc_off,
                  const int* __restrict__ exc_j, const double* __restrict__ exc_scale,
                  const int2* __restrict__ exc_tiles, int n_pad, double* __restrict__ partial, CgStop stop) {
    if (stop.stopped()) return;
    extern __shared__ __align__(16) unsigned char smem[];
    const int NA = BT * 32, warps = BT / 2;
    Rec64 T;
    T.xy = reinterpret_cast<double2*>(smem);
    T.zx = T.xy + NA;
    T.yz = T.zx + NA;
    T.qt = T.yz + NA;
    T.c = reinterpret_cast<double*>(T.qt + NA);
    double4* s_geo = reinterpret_cast<double4*>(T.c + NA);
    double* s_acc = reinterpret_cast<double*>(s_geo + warps * 2 * BT);   // [warp][component][NA]: J-side sums

    int p, q;
    band_pair(blockIdx.x, p, q);
    const int s0 = 32 * blockIdx.y / gridDim.y, s1 = 32 * (blockIdx.y + 1) / gridDim.y;
    const int bands = (P.n_tiles + BT - 1) / BT;
    partial += (size_t)blockIdx.y * bands * 3 * n_pad;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int k = threadIdx.x; k < NA; k += blockDim.x) {
        const double4 a = posq[q * NA + k], b = jvec[q * NA + k];
        T.xy[k] = make_double2(a.x, a.y);
        T.zx[k] = make_double2(a.z, b.x);
        T.yz[k] = make_double2(b.y, b.z);
        T.qt[k] = make_double2(a.w, b.w);
        T.c[k] = 1.0 / (b.w * b.w * b.w);
    }
    for (int k = threadIdx.x; k < warps * 3 * NA; k += blockDim.x) s_acc[k] = 0.0;

    // The warp's 2 x BT tile-pair geometries, one per lane: the whole-box image
    // of the tile pair and its flags.
    const int I0 = p * BT + 2 * warp;
    {
        const int I = I0 + lane / BT, J = q * BT + lane % BT;
        if (lane < 2 * BT) {
            double4 s = make_double4(0, 0, 0, 0);
            unsigned fl = 0u;
            if (I < P.n_tiles && J < P.n_tiles) {
                const double4 cA = tctr[I], cB = tctr[J];
                const TileGeom g = tile_geom(P, (double)P.damp_r2, cA, text[I], cB, text[J]);
                s.x = (cB.x - cA.x) - g.dcx;
                s.y = (cB.y - cA.y) - g.dcy;
                s.z = (cB.z - cA.z) - g.dcz;
                fl = g.fmask | (g.fold ? 8u : 0u) | (g.near ? 16u : 0u);
            }
            s.w = __hiloint2double(0, (int)fl);
            s_geo[warp * 2 * BT + lane] = s;
        }
    }
    double v[2][3];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int I = I0 + k;
        const double4 b = I < P.n_tiles ? jvec[I * 32 + lane] : make_double4(0, 0, 0, 0);
        v[k][0] = b.x;
        v[k][1] = b.y;
        v[k][2] = b.z;
    }
    __syncthreads();
    double f[2][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
    double* acc = s_acc + warp * 3 * NA;
    for (int t = 0; t < BT; t++) {
        const int J = q * BT + t, jbase = J * 32;
        if (J >= P.n_tiles || I0 > J || I0 >= P.n_tiles) continue;
        // What a walk needs of the I atoms beside their operands is read anew
        // for each J tile (L1), so that it takes no registers in between.
        double o[2][3], qi[2], ti[2], c3[2];
        unsigned mk[2], fl = 0u;
        bool masked = false;
        const unsigned real = J == P.n_tiles - 1 && (P.n & 31) ? (1u << (P.n & 31)) - 1u : ~0u;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int I = I0 + k, i = I * 32 + lane;
            const double4 s = s_geo[(warp * 2 + k) * BT + t];
            const double4 a = I < P.n_tiles ? posq[i] : make_double4(0, 0, 0, 0);
            o[k][0] = a.x + s.x;
            o[k][1] = a.y + s.y;
            o[k][2] = a.z + s.z;
            qi[k] = a.w;
            ti[k] = I < P.n_tiles ? jvec[i].w : 0.0;
            c3[k] = 1.0 / (ti[k] * ti[k] * ti[k]);
            fl |= (unsigned)__double2loint(s.w);
            mk[k] = I <= J && i < P.n ? real : 0u;
            if (I == J) mk[k] &= ~((2u << lane) - 1u);   // each pair of a diagonal tile once: j > i
            if (I < P.n_tiles && i < P.n) {
                const int2 et = exc_tiles[I];
                if (J >= et.x && J <= et.y)
                    for (int e = exc_off[i]; e < exc_off[i + 1]; e++) {
                        const unsigned off = (unsigned)(exc_j[e] - jbase);
                        if (off < 32u && exc_scale[e] != 1.0) mk[k] &= ~(1u << off);
                    }
            }
            masked = masked || mk[k] != ~0u;
        }
        double g[3] = {0.0, 0.0, 0.0};
        const int j0 = t * 32;
#define TDP_FWALK64(F, D, M) field_walk64<KIND, F, D, M>(P, T, lane, j0, o, v, qi, ti, c3, mk, fl, s0, s1, f, g)
        if (__any_sync(kFull, masked)) {
            TDP_FWALK64(true, true, true);
        } else if (fl & 8u) {
            if (fl & 16u) TDP_FWALK64(true, true, false);
            else TDP_FWALK64(true, false, false);
        } else if (fl & 16u) {
            TDP_FWALK64(false, true, false);
        } else {
            TDP_FWALK64(false, false, false);
        }
#undef TDP_FWALK64
        const int jl = j0 + ((lane + s1) & 31);   // the J atom whose sums the lane holds now
#pragma unroll
        for (int c = 0; c < 3; c++) acc[c * NA + jl] += g[c];
        __syncwarp();
    }
    // I-side sums: slot q of band p; on the diagonal band they join the J-side
    // sums of the same atoms.
#pragma unroll
    for (int k = 0; k < 2; k++) {
        if (I0 + k >= P.n_tiles) continue;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            if (p == q) acc[c * NA + (2 * warp + k) * 32 + lane] += f[k][c];
            else partial[((size_t)q * 3 + c) * n_pad + (I0 + k) * 32 + lane] = f[k][c];
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < NA; k += blockDim.x)
#pragma unroll
        for (int c = 0; c < 3; c++) {
            double s = 0.0;
            for (int w = 0; w < warps; w++) s += s_acc[(w * 3 + c) * NA + k];
            partial[((size_t)p * 3 + c) * n_pad + q * NA + k] = s;
        }
}

// Plain form: an atom's slots, in slot order, into slot 0, and its partner
// pairs.  A CTA takes 32 atoms: warp c adds component c's slots (coalesced), and
// the three warps share the partners.
template <int KIND>
__global__ void __launch_bounds__(96)
    k_field_slots(PairParams P, int fused, const double4* __restrict__ posq, const double4* __restrict__ jvec,
                  const double4* __restrict__ lab, const double* __restrict__ pos, const int* __restrict__ exc_off,
                  const int* __restrict__ exc_j, const double* __restrict__ exc_m, const double* __restrict__ exc_s,
                  int n_pad, int nslot, double* __restrict__ partial, CgStop stop) {
    if (stop.stopped()) return;
    __shared__ double s_part[3][3][32];
    const int lane = threadIdx.x & 31, c = threadIdx.x >> 5, k = blockIdx.x * 32 + lane;
    double f[3] = {0.0, 0.0, 0.0};
    if (k < P.n) {
        const double ti = jvec[k].w;
        for (int e = exc_off[k] + c; e < exc_off[k + 1]; e += 3)
            add_partner<KIND>(P, fused, posq, jvec, lab, pos, exc_j, exc_m, exc_s, k, e, ti, f);
    }
#pragma unroll
    for (int d = 0; d < 3; d++) s_part[c][d][lane] = f[d];
    __syncthreads();
    const size_t count = (size_t)3 * n_pad;
    double* out = partial + (size_t)c * n_pad + k;
    double s = 0.0;
#pragma unroll 8
    for (int j = 0; j < nslot; j++) s += out[j * count];
    *out = s + s_part[0][c][lane] + s_part[1][c][lane] + s_part[2][c][lane];
}

// ---------------------------------------------------------------------------
// One CG iteration after its matvec, in one launch: a cluster of eight CTAs
// holds every atom's p, r and q in registers between the two scalar products,
// which cross it through distributed shared memory in a fixed order.  Bound by
// latency (launch, two cluster barriers, a chain of loads), as the four
// launches before it were (sums, q, update, p: 4.4 + 4.2 + 5.3 + 5.1 us at 648
// atoms, 6.1 + 4.7 + 5.3 + 4.9 at 12,288, and a gap after each).  With the
// epsilon through pinned memory and the next iteration queued ahead, an
// evaluation went from 436 to 270 us at 648 atoms (mixed), 555 to 453 at 1,029
// and 5111 to 5033 at 12,288 (FP64), 2369 to 2267 at 12,288 (mixed).
// ---------------------------------------------------------------------------
constexpr int kCgCtas = 8, kCgThreads = 512, kCgCap = kCgCtas * kCgThreads;

// The sum over the cluster of a and b, the same in every thread.  buf: two
// doubles per warp and two for the CTA, used once per launch.
__device__ __forceinline__ void cluster_sum2(cg::cluster_group& cl, double& a, double& b, double (&buf)[2][17]) {
    a = warp_sum(a);
    b = warp_sum(b);
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        buf[0][w] = a;
        buf[1][w] = b;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        double t = 0.0;
        for (int k = 0; k < (int)blockDim.x / 32; k++) t += buf[threadIdx.x][k];
        buf[threadIdx.x][16] = t;
    }
    cl.sync();
    a = b = 0.0;
#pragma unroll
    for (int c = 0; c < kCgCtas; c++) {
        a += *cl.map_shared_rank(&buf[0][16], c);
        b += *cl.map_shared_rank(&buf[1][16], c);
    }
}

struct CgArrays {
    const int* order;
    const double *partial, *salpha, *thole, *E;
    double *y, *r, *p, *scal_rr, *scal_eps, *host_eps;
    unsigned long long* acc;   // mixed form: the matvec's fixed-point sums, else null
    double inv_scale;
    int n, n_pad, slot;        // reads scal[slot], writes scal[slot + 1]
    CgStop stop;
};

// q = p - S T S p, a = r.r / p.q, y += a p, r -= a q, p = r + (r'.r' / r.r) p and
// the next operand S p.  DONE: the matvec's sums still lie in the fixed-point
// accumulator, and the thread of slot k also evaluates its partner pairs, as
// k_field_done does.
template <class R, bool DONE, int M>
__global__ void __cluster_dims__(kCgCtas, 1, 1) __launch_bounds__(kCgThreads)
    k_cg_step(PairParams P, CgArrays A, const typename Vec4T<R>::type* __restrict__ posq,
              typename Vec4T<R>::type* vec, const double* __restrict__ pos, const int* __restrict__ exc_off,
              const int* __restrict__ exc_j, const double* __restrict__ exc_m, const double* __restrict__ exc_s) {
    __shared__ double buf[2][2][17];
    cg::cluster_group cl = cg::this_cluster();
    const int k0 = blockIdx.x * blockDim.x + threadIdx.x;
    const bool stopped = A.stop.stopped();
    d3 t[M], p[M], r[M];
    double s[M], pq = 0.0, zero = 0.0;
    int id[M];
#pragma unroll
    for (int m = 0; m < M; m++) {
        const int k = k0 + m * kCgCap;
        id[m] = -1;
        double f[3] = {0.0, 0.0, 0.0};
        if (DONE) {
            if (k < A.n_pad)
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    f[c] = (double)(long long)A.acc[(size_t)c * A.n_pad + k] * A.inv_scale;
                    A.acc[(size_t)c * A.n_pad + k] = 0ull;
                }
        }
        if (k >= A.n || stopped) continue;
        const int i = id[m] = A.order[k];
        if (DONE) {
            const double ti = (double)vec[k].w;
            for (int e = exc_off[k]; e < exc_off[k + 1]; e++)
                add_partner<1>(P, 0, posq, (const typename Vec4T<R>::type*)vec, (const typename Vec4T<R>::type*)nullptr,
                               pos, exc_j, exc_m, exc_s, k, e, ti, f);
        } else {
#pragma unroll
            for (int c = 0; c < 3; c++) f[c] = A.partial[(size_t)c * A.n_pad + k];
        }
        s[m] = A.salpha[i];
        p[m] = ld3(A.p + 3 * (size_t)i);
        r[m] = ld3(A.r + 3 * (size_t)i);
        t[m] = p[m] - d3{f[0], f[1], f[2]} * s[m];   // q
        pq += dot(p[m], t[m]);
    }
    if (stopped) return;   // the same in every CTA
    cluster_sum2(cl, pq, zero, buf[0]);
    const double rr = A.scal_rr[A.slot], a = rr / pq;
    double rn = 0.0, en = 0.0;
#pragma unroll
    for (int m = 0; m < M; m++) {
        if (id[m] < 0) continue;
        double* y = A.y + 3 * (size_t)id[m];
        const d3 yv = ld3(y) + p[m] * a;
        y[0] = yv.x;
        y[1] = yv.y;
        y[2] = yv.z;
        r[m] = r[m] - t[m] * a;
        double* ro = A.r + 3 * (size_t)id[m];
        ro[0] = r[m].x;
        ro[1] = r[m].y;
        ro[2] = r[m].z;
        const double v = dot(r[m], r[m]);
        rn += v;
        en += s[m] * s[m] * v;
    }
    cluster_sum2(cl, rn, en, buf[1]);
    if (k0 == 0) {
        const double eps = sqrt(en / (double)A.n);
        A.scal_rr[A.slot + 1] = rn;
        A.scal_eps[A.slot + 1] = eps;
        *(volatile double*)A.host_eps = eps;
    }
    const double beta = rn / rr;
#pragma unroll
    for (int m = 0; m < M; m++) {
        if (id[m] < 0) continue;
        const int i = id[m];
        const d3 pv = r[m] + p[m] * beta;
        double* po = A.p + 3 * (size_t)i;
        po[0] = pv.x;
        po[1] = pv.y;
        po[2] = pv.z;
        store_operand<R>(vec, k0 + m * kCgCap, pv * s[m], A.thole[i]);
    }
    cl.sync();   // no CTA leaves while another reads its sums
}

// The residual of y: r = p = S (E + T mu) - y (use_partial 0: E holds the field
// already), the operand S p and the scalars of `slot`.
template <class R, int M>
__global__ void __cluster_dims__(kCgCtas, 1, 1) __launch_bounds__(kCgThreads)
    k_cg_start(CgArrays A, typename Vec4T<R>::type* __restrict__ vec, int use_partial) {
    __shared__ double buf[2][17];
    cg::cluster_group cl = cg::this_cluster();
    const int k0 = blockIdx.x * blockDim.x + threadIdx.x;
    double rr = 0.0, ee = 0.0;
#pragma unroll
    for (int m = 0; m < M; m++) {
        const int k = k0 + m * kCgCap;
        if (k >= A.n) continue;
        const int i = A.order[k];
        d3 e = ld3(A.E + 3 * (size_t)i);
        if (use_partial) e = e + d3{A.partial[k], A.partial[A.n_pad + k], A.partial[2 * (size_t)A.n_pad + k]};
        const double s = A.salpha[i];
        const d3 rv = e * s - ld3(A.y + 3 * (size_t)i);
        double *r = A.r + 3 * (size_t)i, *p = A.p + 3 * (size_t)i;
        r[0] = p[0] = rv.x;
        r[1] = p[1] = rv.y;
        r[2] = p[2] = rv.z;
        store_operand<R>(vec, k, rv * s, A.thole[i]);
        const double v = dot(rv, rv);
        rr += v;
        ee += s * s * v;
    }
    cluster_sum2(cl, rr, ee, buf);
    if (k0 == 0) {
        const double eps = sqrt(ee / (double)A.n);
        A.scal_rr[A.slot] = rr;
        A.scal_eps[A.slot] = eps;
        *(volatile double*)A.host_eps = eps;
    }
    cl.sync();
}

// ---------------------------------------------------------------------------
// Energy / force / torque kernel (index order: within a tile pair I < J every
// lane's atom has the lower index, the reference's orientation I = lower).
// ---------------------------------------------------------------------------
template <class R>
__device__ __forceinline__ EAtom<R> eatom(typename Vec4T<R>::type pq, typename Vec4T<R>::type d,
                                          typename Vec4T<R>::type u) {
    EAtom<R> a;
    a.q = pq.w;
    a.mx = d.x;
    a.my = d.y;
    a.mz = d.z;
    a.t = d.w;
    a.ux = u.x;
    a.uy = u.y;
    a.uz = u.z;
    return a;
}

// formQIRotationMatrix's test on the raw positions, pI.y != pK.y || pI.z !=
// pK.z (RTDF.cpp:584): displacements above 1e-5 nm decide it; below that the
// raw FP64 coordinates are compared.
template <class R>
__device__ __forceinline__ bool yz_differ(R dy, R dz, const double2* __restrict__ yz, int i, int j, int nmax) {
    bool d = fabs(dy) > R(1e-5) || fabs(dz) > R(1e-5);
    if (!d) {
        const double2 a = yz[min(i, nmax)], b = yz[min(j, nmax)];
        d = (a.x != b.x) || (a.y != b.y);
    }
    return d;
}

// J records of the plain energy kernel in pieces (see Rec64).
struct ERec64 {
    double2 *xy, *zq, *mm, *mu, *uu;   // (x, y), (z, q), (mx, my), (mz, ux), (uy, uz)
    double* t;
    __device__ __forceinline__ ERec64(double2* s, int n)
        : xy(s), zq(s + n), mm(s + 2 * n), mu(s + 3 * n), uu(s + 4 * n), t(reinterpret_cast<double*>(s + 5 * n)) {}
    __device__ __forceinline__ EAtom<double> atom(int k) const {
        EAtom<double> a;
        const double2 m = mm[k], x = mu[k], u = uu[k];
        a.q = zq[k].y;
        a.mx = m.x;
        a.my = m.y;
        a.mz = x.x;
        a.ux = x.y;
        a.uy = u.x;
        a.uz = u.y;
        a.t = t[k];
        return a;
    }
};

// LAB (non-SLOW tile pairs beyond the damping range only): pair_energy_lab.
template <bool FOLD, bool SLOW, bool LAB = false>
__device__ __forceinline__ void energy_walk(const PairParams& P, const double2* __restrict__ yz, const ERec64& T, int j0,
                                            int lane, int i, int jbase, double oix, double oiy, double oiz,
                                            const EAtom<double>& me, bool diag, unsigned partners, unsigned fold,
                                            double f[6], double g[6], double& en) {
    const int nxt = (lane + 1) & 31;
    const int nmax = P.n_tiles * 32 - 1;
    // LAB: the walk sums V_ij (I side) and V_ji (J side, rotating with the
    // J atoms) and turns them into torques once at the end (pair_energy_lab).
    double vi[3] = {0, 0, 0}, vj[3] = {0, 0, 0};
    const double Pi[3] = {me.mx + me.ux, me.my + me.uy, me.mz + me.uz}, ui[3] = {me.ux, me.uy, me.uz};
    const double kap = P.mutual ? 1.0 : -1.0;
#pragma unroll 1
    for (int s = 0; s < 32; s++) {
        const int jj = (lane + s) & 31;
        const int j = jbase + jj;
        const double2 pxy = T.xy[j0 + jj], pzq = T.zq[j0 + jj];
        double dx, dy, dz;
        pair_delta<FOLD>(P, fold, pxy.x, pxy.y, pzq.x, oix, oiy, oiz, dx, dy, dz);
        if constexpr (LAB) {
            const double2 mm = T.mm[j0 + jj], mu = T.mu[j0 + jj], uu = T.uu[j0 + jj];
            const double w[3] = {mu.y, uu.x, uu.y}, Q[3] = {mm.x + w[0], mm.y + w[1], mu.x + w[2]};
            pair_energy_lab(dx, dy, dz, me.q, Pi, ui, pzq.y, Q, w, kap,
                            [&] { return yz_differ<double>(dy, dz, yz, i, j, nmax); }, f, g, vi, vj, en);
#pragma unroll
            for (int c = 0; c < 3; c++) {
                g[c] = __shfl_sync(kFull, g[c], nxt);
                vj[c] = __shfl_sync(kFull, vj[c], nxt);
            }
        } else {
            const double damp_r2 = (double)P.damp_r2, rv4p = (double)P.rinv4_power, rv4f = (double)P.rinv4_fill;
            double r2 = dx * dx + dy * dy + dz * dz;
            if (SLOW && skip_pair(s, lane, i, j, P.n, partners, jj, diag)) r2 = (double)INFINITY;
            const bool yzd = yz_differ<double>(dy, dz, yz, i, j, nmax);
            const EAtom<double> other = T.atom(j0 + jj);
            if (!SLOW || !diag) {
                pair_energy_sides<double, 3>(dx, dy, dz, r2, yzd, me, other, 1.0, 1.0, damp_r2, rv4p, rv4f,
                                             P.mutual != 0, f[0], f[1], f[2], f[3], f[4], f[5], g[0], g[1], g[2], g[3],
                                             g[4], g[5], en);
            } else {
                // Diagonal tile: the lane's atom is the lower index iff lane + s < 32.
                const bool lo = lane + s < 32;
                const EAtom<double> A = lo ? me : other;
                const EAtom<double> B = lo ? other : me;
                const double sg = lo ? 1.0 : -1.0;
                double a[6] = {0, 0, 0, 0, 0, 0}, b[6] = {0, 0, 0, 0, 0, 0};
                pair_energy_sides<double, 3>(sg * dx, sg * dy, sg * dz, r2, yzd, A, B, 1.0, 1.0, damp_r2, rv4p, rv4f,
                                             P.mutual != 0, a[0], a[1], a[2], a[3], a[4], a[5], b[0], b[1], b[2],
                                             b[3], b[4], b[5], en);
#pragma unroll
                for (int c = 0; c < 6; c++) {
                    f[c] += lo ? a[c] : b[c];
                    g[c] += lo ? b[c] : a[c];
                }
            }
#pragma unroll
            for (int c = 0; c < 6; c++) g[c] = __shfl_sync(kFull, g[c], nxt);
        }
    }
    if (LAB) {
        // tau = -perm(m x sum V) and the dipole energy 0.5 m.sum V: the lane's
        // I atom, and J atom jbase + lane.
        const EAtom<double> mj = T.atom(j0 + lane);
        en += 0.5 * (me.mx * vi[0] + me.my * vi[1] + me.mz * vi[2] + mj.mx * vj[0] + mj.my * vj[1] + mj.mz * vj[2]);
        f[3] -= me.mz * vi[0] - me.mx * vi[2];
        f[4] -= me.mx * vi[1] - me.my * vi[0];
        f[5] -= me.my * vi[2] - me.mz * vi[1];
        g[3] -= mj.mz * vj[0] - mj.mx * vj[2];
        g[4] -= mj.mx * vj[1] - mj.my * vj[0];
        g[5] -= mj.my * vj[2] - mj.mz * vj[1];
    }
}

// ---------------------------------------------------------------------------
// Mixed-form energy / force / torque walk: the lane's I atom against J atoms m
// and m + 16 of the tile at once (m = (lane + s) & 15) in f32x2 halves, the
// J-side sums riding packed and rotating one lane per step as in the field
// walks.
//
// Orientation.  The reference's pair routine has I = lower index, K = higher,
// d = p_K - p_I.  Tiles here are in spatial order, so a pair may come with its
// roles exchanged.  That flips Z and Y of the quasi-internal frame (a rotation
// by pi about X, under which every vector expression of the routine is
// covariant) and leaves X; what remains is that the terms linear in a charge
// change sign, and the sign of the force.  So a pair whose I atom has the
// higher index is evaluated with both charges negated (their product is not)
// and the force negated: the sign bit of (index of J - index of I) xor-ed in.
//
// MODE 0, 1: the pair routine (RTDF.cpp:129-366) in the lab frame, for unit
// scales and rInvVec[4] = 0 (the default, see TDP_FLAG_DD_FORCE_R4).  What is
// left of the quasi-internal frame is its X row, the axis its multipole
// algebra treats as the bond axis (component 0); with x = a u^3, e = exp(-x),
// tc = 1 - e, w = 1 - (1 + x) e, t0 = 1 - (1 + 3x/2) e, l = 2 (Mutual) or 0:
//   V_ij  = (q_j/r^2 - 3 (m_j0 + w u_j0)/r^3) X + (m_j + tc u_j)/r^3
//   V_ji  = (-q_i/r^2 - 3 (m_i0 + w u_i0)/r^3) X + (m_i + tc u_i)/r^3
//   Vd_ij = (tc q_j/r^2 - 3 w (m_j0 + l u_j0)/r^3) X + tc (m_j + l u_j)/r^3, Vd_ji alike
//   S   = m_i x V_ij + m_j x V_ji + u_i x Vd_ij + u_j x Vd_ji
//   f   = (S x X)/r + (q_i q_j/r^2 - 2 (q_i m_j0 - q_j m_i0 + t0 (q_i u_j0 - q_j u_i0))/r^3) X
//   E   = q_i q_j/r + (q_j m_i0 - q_i m_j0 + tc (q_j u_i0 - q_i u_j0))/(2 r^2) + (m_i.V_ij + m_j.V_ji)/2
//   F_I -= perm(f), F_J += perm(f), tau_I = -perm(m_i x V_ij), tau_J = -perm(m_j x V_ji)
// with perm(v) = (v_y, v_z, v_x), the reference's permuted back rotation
// (:150-159).  The parts of S without X cancel pairwise, so S = K x X with
// K = a m_i + b m_j + c u_i + d u_j (a, b, c, d the X coefficients of V_ij,
// V_ji, Vd_ij, Vd_ji) and S x X = (K.X) X - K.  Torques and the dipole energy
// are linear in V with an atom's own dipole fixed: the walk sums V and the
// caller takes one cross and one dot product per atom.  MODE 0 is the walk of
// tile pairs that no damping reaches (tc = w = t0 = 1): with P = m + u and
// k = l - 1, K = a P_i + b P_j + g u_j0 u_i + g u_i0 u_j, g = -3 k/r^3.
// X is (d_y^2 + d_z^2, -d_x d_y, -d_x d_z)/(r sqrt(d_y^2 + d_z^2)) where the
// pair's y or z coordinates differ (:584); pairs within 1e-5 nm of the x axis
// take the reference's test and Gram-Schmidt as is.
// MODE 2: the quasi-internal frame routine itself (TDP_FLAG_DD_FORCE_R4).
// ---------------------------------------------------------------------------
struct EItemTile {
    float4 p0[16], p1[16];   // (x, x', y, y'), (z, z', q, q')   (' = atom m + 16)
    float4 d0[16], d1[16];   // (dx, dx', dy, dy'), (dz, dz', t, t'): m, or m + u in MODE 0
    float4 u0[16], u1[16];   // (ux, ux', uy, uy'), (uz, uz', 1/t, 1/t')
    int2 id[16];             // atom indices
};

// FP64 positions of the J tile (open systems' charge energy).
struct EItemPos {
    double x[32], y[32], z[32];
};

__device__ __forceinline__ void stage_eitem(EItemTile& T, int lane, float4 p, float4 d, float4 u, int id) {
    const int m = lane & 15, h = lane >> 4;
    float* p0 = reinterpret_cast<float*>(&T.p0[m]);
    float* p1 = reinterpret_cast<float*>(&T.p1[m]);
    float* d0 = reinterpret_cast<float*>(&T.d0[m]);
    float* d1 = reinterpret_cast<float*>(&T.d1[m]);
    float* u0 = reinterpret_cast<float*>(&T.u0[m]);
    float* u1 = reinterpret_cast<float*>(&T.u1[m]);
    p0[h] = p.x;
    p0[2 + h] = p.y;
    p1[h] = p.z;
    p1[2 + h] = p.w;
    d0[h] = d.x;
    d0[2 + h] = d.y;
    d1[h] = d.z;
    d1[2 + h] = d.w;
    u0[h] = u.x;
    u0[2 + h] = u.y;
    u1[h] = u.z;
    u1[2 + h] = 1.0f / d.w;
    reinterpret_cast<int*>(&T.id[m])[h] = id;
}

__device__ __forceinline__ f2 xneg2(f2 a) { return a ^ 0x8000000080000000ull; }

// X row of formQIRotationMatrix (RTDF.cpp:580-593) for one pair, as the
// general walk forms it.
__device__ __forceinline__ void qi_frame_x(float dx, float dy, float dz, float rinv, bool yzd, float& xx, float& xy,
                                           float& xz) {
    const float zx = dx * rinv, zy = dy * rinv, zz = dz * rinv;
    xx = zx + (yzd ? 1.0f : 0.0f);
    xy = zy + (yzd ? 0.0f : 1.0f);
    xz = zz;
    const float dt = zx * xx + zy * xy + zz * xz;
    xx -= zx * dt;
    xy -= zy * dt;
    xz -= zz * dt;
    const float n2 = xx * xx + xy * xy + xz * xz;
    const float s = n2 > 0.0f ? rsqrtf(n2) : 1.0f;
    xx *= s;
    xy *= s;
    xz *= s;
}

// formQIRotationMatrix's test on the raw positions by slot, pI.y != pK.y ||
// pI.z != pK.z (RTDF.cpp:584): displacements above 1e-5 nm decide it; below
// that the raw FP64 coordinates are compared.
__device__ __forceinline__ bool yz_differ_slot(float dy, float dz, const double* __restrict__ pos, int i, int j) {
    if (fabsf(dy) > 1e-5f || fabsf(dz) > 1e-5f) return true;
    return pos[3 * (size_t)i + 1] != pos[3 * (size_t)j + 1] || pos[3 * (size_t)i + 2] != pos[3 * (size_t)j + 2];
}

// The index-order records of the atoms (FP32 offsets from the centres of the
// 32-atom tiles in index order), and the sorted ones by slot.
struct IndexRecords {
    const float4* posq;
    const double4* tctr;
    const float4 *posq_s, *dipt_s, *ind_s;
};

// p_j - p_i of slots i and j (atoms id_i, id_j) from the index-order records,
// whose rounding does not change when the atoms are sorted anew.
__device__ __forceinline__ void index_delta(const PairParams& P, const IndexRecords& R, const double* __restrict__ pos,
                                            int i, int j, int id_i, int id_j, float& dx, float& dy, float& dz) {
    const bool swap = id_i > id_j;
    const int lo = swap ? id_j : id_i, hi = swap ? id_i : id_j;
    const float4 a = R.posq[lo], b = R.posq[hi];
    const double4 ca = R.tctr[lo >> 5], cb = R.tctr[hi >> 5];
    double c[3] = {cb.x - ca.x, cb.y - ca.y, cb.z - ca.z};
    const float pa[3] = {a.x, a.y, a.z}, pb[3] = {b.x, b.y, b.z};
    float d[3];
    bool near_half = false;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        if (P.periodic) c[k] = fold_d(c[k], P.box[k], P.inv_box[k]);
        d[k] = pb[k] - (pa[k] - (float)c[k]);
        if (P.periodic) {
            d[k] = fold_f(d[k], (float)P.box[k], (float)P.inv_box[k]);
            near_half = near_half || fabsf(d[k]) >= (float)P.half_box_tol[k];
        }
    }
    if (near_half) {
        const d3 e = exact_delta(P, pos, swap ? j : i, swap ? i : j);
        d[0] = (float)e.x;
        d[1] = (float)e.y;
        d[2] = (float)e.z;
    }
    dx = swap ? -d[0] : d[0];
    dy = swap ? -d[1] : d[1];
    dz = swap ? -d[2] : d[2];
}

// The pair routine in its quasi-internal frame (RTDF.cpp:129-366) on both
// halves, given the frame's X row: -f (added to I's force, subtracted from
// K's), the vectors that come off the two torques, and twice the energy.
struct QiPair {
    f2 nfx, nfy, nfz, tx, ty, tz, ux, uy, uz, e2;
};

__device__ __forceinline__ QiPair qi_pair2(const PairParams& P, f2 DX, f2 DY, f2 DZ, f2 R2, f2 RINV, float r2a,
                                           float r2b, f2 XX, f2 XY, f2 XZ, f2 QIS, f2 MIX, f2 MIY, f2 MIZ, f2 UIX,
                                           f2 UIY, f2 UIZ, float ti, float iti, f2 QJS, f2 MJX, f2 MJY, f2 MJZ, f2 UJX,
                                           f2 UJY, f2 UJZ, float tja, float tjb, float itja, float itjb) {
    const f2 RV4P = bc2(P.rinv4_power), RV4F = bc2(P.rinv4_fill), ITI = bc2(iti), ONE = bc2(1.0f);
    const float damp_r2 = P.damp_r2;
    // QI frame: Z along d, Y = Z x X.
    const f2 ZX = mul2(DX, RINV), ZY = mul2(DY, RINV), ZZ = mul2(DZ, RINV);
    const f2 YX = fma2(ZY, XZ, neg2(mul2(ZZ, XY)));
    const f2 YY = fma2(ZZ, XX, neg2(mul2(ZX, XZ)));
    const f2 YZ = fma2(ZX, XY, neg2(mul2(ZY, XX)));
    // Rotated multipoles.
    const f2 uI0 = dot2(XX, XY, XZ, UIX, UIY, UIZ), uI1 = dot2(YX, YY, YZ, UIX, UIY, UIZ),
             uI2 = dot2(ZX, ZY, ZZ, UIX, UIY, UIZ);
    const f2 uJ0 = dot2(XX, XY, XZ, UJX, UJY, UJZ), uJ1 = dot2(YX, YY, YZ, UJX, UJY, UJZ),
             uJ2 = dot2(ZX, ZY, ZZ, UJX, UJY, UJZ);
            const f2 QI1 = dot2(XX, XY, XZ, MIX, MIY, MIZ), QI2 = dot2(YX, YY, YZ, MIX, MIY, MIZ),
             QI3 = dot2(ZX, ZY, ZZ, MIX, MIY, MIZ);
    const f2 QJ1 = dot2(XX, XY, XZ, MJX, MJY, MJZ), QJ2 = dot2(YX, YY, YZ, MJX, MJY, MJZ),
             QJ3 = dot2(ZX, ZY, ZZ, MJX, MJY, MJZ);
    const f2 rv1 = RINV, rv2 = mul2(RINV, RINV), rv3 = mul2(rv2, RINV);
    const f2 rv4 = fma2(RV4P, mul2(rv3, RINV), RV4F);
    // Thole factors (1 beyond damp_r2 or where t_i t_j <= 1e-5, as the reference).
    f2 tc = ONE, td0 = ONE, td1 = ONE, dtc = ONE, dtd0 = ONE, dtd1 = ONE;
    if (r2a < damp_r2 || r2b < damp_r2) {
        const f2 R = mul2(R2, RINV);
        const f2 U = mul2(mul2(R, ITI), pk2(itja, itjb));
        const f2 AM = pk2(fminf(ti, tja), fminf(ti, tjb));
        const f2 AU3 = mul2(AM, mul2(U, mul2(U, U)));
        float xa, xb;
        un2(AU3, xa, xb);
        const bool da = r2a < damp_r2 && fabsf(ti * tja) > 1.0e-5f;
        const bool db = r2b < damp_r2 && fabsf(ti * tjb) > 1.0e-5f;
        const f2 EX = pk2(da ? __expf(-xa) : 0.0f, db ? __expf(-xb) : 0.0f);
        const f2 AUs = pk2(da ? xa : 0.0f, db ? xb : 0.0f);   // no inf/NaN into the products
        const f2 NEX = neg2(EX);
        tc = add2(ONE, NEX);
        td1 = tc;
        td0 = fma2(NEX, fma2(bc2(1.5f), AUs, ONE), ONE);
        dtc = td0;
        dtd0 = fma2(NEX, fma2(mul2(bc2(1.5f), AUs), AUs, add2(ONE, AUs)), ONE);
        dtd1 = fma2(NEX, add2(ONE, AUs), ONE);
    }
    // Interaction terms (mS = iS = 1).
    f2 eP = rv1, dP = mul2(bc2(-0.5f), rv2);
    f2 Vij0 = mul2(eP, QJS), Vji0 = mul2(eP, QIS), VijR0 = mul2(dP, QJS), VjiR0 = mul2(dP, QIS);
    eP = rv2;
    f2 eU = mul2(rv2, tc);
    dP = neg2(rv3);
    f2 dU = mul2(mul2(bc2(-2.0f), rv3), dtc);
    Vij0 = sub2(Vij0, fma2(eP, QJ1, mul2(eU, uJ0)));
    const f2 Vji1n = mul2(eP, QIS);   // -Vji1 so far (subtracted below: exact)
    VijR0 = sub2(VijR0, fma2(dP, QJ1, mul2(dU, uJ0)));
    f2 VjiR1 = mul2(rv3, QIS);        // -(dP QIS), dP = -rv3: exact
    f2 Vjid0 = neg2(mul2(eU, QIS));
    f2 Vij1 = mul2(eP, QJS);
    Vji0 = add2(Vji0, fma2(eP, QI1, mul2(eU, uI0)));
    f2 VijR1 = mul2(dP, QJS);
    VjiR0 = add2(VjiR0, fma2(dP, QI1, mul2(dU, uI0)));
    f2 Vijd0 = mul2(eU, QJS);
    eP = mul2(bc2(-2.0f), rv3);
    eU = mul2(eP, td0);
    dP = mul2(bc2(3.0f), rv4);
    dU = mul2(mul2(bc2(6.0f), rv4), dtd0);
    Vij1 = add2(Vij1, fma2(eP, QJ1, mul2(eU, uJ0)));
    f2 Vji1 = sub2(fma2(eP, QI1, mul2(eU, uI0)), Vji1n);
    VijR1 = add2(VijR1, fma2(dP, QJ1, mul2(dU, uJ0)));
    VjiR1 = add2(VjiR1, fma2(dP, QI1, mul2(dU, uI0)));
    Vijd0 = fma2(eU, QJ1, Vijd0);
    Vjid0 = fma2(eU, QI1, Vjid0);
    eP = rv3;
    eU = mul2(rv3, td1);
    dP = mul2(bc2(-1.5f), rv4);
    dU = mul2(mul2(bc2(-3.0f), rv4), dtd1);
    const f2 Vij2 = fma2(eP, QJ2, mul2(eU, uJ1)), Vji2 = fma2(eP, QI2, mul2(eU, uI1));
    const f2 VijR2 = fma2(dP, QJ2, mul2(dU, uJ1)), VjiR2 = fma2(dP, QI2, mul2(dU, uI1));
    const f2 Vijd1 = mul2(eU, QJ2), Vjid1 = mul2(eU, QI2);
    const f2 Vij3 = fma2(eP, QJ3, mul2(eU, uJ2)), Vji3 = fma2(eP, QI3, mul2(eU, uI2));
    const f2 VijR3 = fma2(dP, QJ3, mul2(dU, uJ2)), VjiR3 = fma2(dP, QI3, mul2(dU, uI2));
    const f2 Vijd2 = mul2(eU, QJ3), Vjid2 = mul2(eU, QI3);

    f2 fIZ = fma2(QIS, VijR0, fma2(QI1, VijR1, fma2(QI2, VijR2, mul2(QI3, VijR3))));
    f2 fJZ = fma2(QJS, VjiR0, fma2(QJ1, VjiR1, fma2(QJ2, VjiR2, mul2(QJ3, VjiR3))));
    const f2 EIX = sub2(mul2(QI3, Vij1), mul2(QI1, Vij3));
    const f2 EIY = sub2(mul2(QI1, Vij2), mul2(QI2, Vij1));
    const f2 EJX = sub2(mul2(QJ3, Vji1), mul2(QJ1, Vji3));
    const f2 EJY = sub2(mul2(QJ1, Vji2), mul2(QJ2, Vji1));
    f2 iEIX = sub2(mul2(uI2, Vijd0), mul2(uI0, Vijd2));
    f2 iEJX = sub2(mul2(uJ2, Vjid0), mul2(uJ0, Vjid2));
    f2 iEIY = sub2(mul2(uI0, Vijd1), mul2(uI1, Vijd0));
    f2 iEJY = sub2(mul2(uJ0, Vjid1), mul2(uJ1, Vjid0));
    if (P.mutual) {
        f2 eC = mul2(mul2(bc2(-4.0f), rv3), td0);
        f2 dC = mul2(mul2(bc2(6.0f), rv4), dtd0);
        iEIX = fma2(mul2(eC, uI2), uJ0, iEIX);
        iEJX = fma2(mul2(eC, uJ2), uI0, iEJX);
        iEIY = sub2(iEIY, mul2(mul2(eC, uI1), uJ0));
        iEJY = sub2(iEJY, mul2(mul2(eC, uJ1), uI0));
        fIZ = fma2(mul2(dC, uI0), uJ0, fIZ);
        fJZ = fma2(mul2(dC, uJ0), uI0, fJZ);
        eC = mul2(mul2(bc2(2.0f), rv3), td1);
        dC = mul2(mul2(bc2(-3.0f), rv4), dtd1);
        iEIX = sub2(iEIX, mul2(mul2(eC, uI0), uJ2));
        iEJX = sub2(iEJX, mul2(mul2(eC, uJ0), uI2));
        iEIY = fma2(mul2(eC, uI0), uJ1, iEIY);
        iEJY = fma2(mul2(eC, uJ0), uI1, iEJY);
        const f2 uu = fma2(uI1, uJ1, mul2(uI2, uJ2));
        fIZ = fma2(dC, uu, fIZ);
        fJZ = fma2(dC, uu, fJZ);
    }
    // nqf = -qf (the QI-frame force); every sign flip below is exact.
    const f2 nqf0 = neg2(mul2(RINV, add2(add2(EIY, EJY), add2(iEIY, iEJY))));
    const f2 nqf1 = mul2(RINV, add2(add2(EIX, EJX), add2(iEIX, iEJX)));
    const f2 nqf2 = add2(fJZ, fIZ);
    // Back rotation with the reference's permuted matrix: nfv = -fv.
    const f2 nfvx = fma2(YY, nqf0, fma2(ZY, nqf1, mul2(XY, nqf2)));
    const f2 nfvy = fma2(YZ, nqf0, fma2(ZZ, nqf1, mul2(XZ, nqf2)));
    const f2 nfvz = fma2(YX, nqf0, fma2(ZX, nqf1, mul2(XX, nqf2)));
    QiPair o;
    o.nfx = nfvx;
    o.nfy = nfvy;
    o.nfz = nfvz;
    const f2 EIZ = sub2(mul2(QI2, Vij3), mul2(QI3, Vij2)), EJZ = sub2(mul2(QJ2, Vji3), mul2(QJ3, Vji2));
    o.tx = fma2(YY, EIX, fma2(ZY, EIY, mul2(XY, EIZ)));
    o.ty = fma2(YZ, EIX, fma2(ZZ, EIY, mul2(XZ, EIZ)));
    o.tz = fma2(YX, EIX, fma2(ZX, EIY, mul2(XX, EIZ)));
    o.ux = fma2(YY, EJX, fma2(ZY, EJY, mul2(XY, EJZ)));
    o.uy = fma2(YZ, EJX, fma2(ZZ, EJY, mul2(XZ, EJZ)));
    o.uz = fma2(YX, EJX, fma2(ZX, EJY, mul2(XX, EJZ)));
    o.e2 = fma2(QI3, Vij3, fma2(QJ3, Vji3, fma2(QI2, Vij2, fma2(QJ2, Vji2, fma2(QI1, Vij1, fma2(QJ1, Vji1,
               fma2(QIS, Vij0, mul2(QJS, Vji0))))))));
    return o;
}

// Pairs this close to the x axis (kNearAxis2, nm^2) and no further apart than
// sqrt(kAxisListRange2) = 1.5 times the damping range go to the list of
// k_axis_pairs.  Further pairs have smaller forces: within kNearAxisFar2 they
// keep the lab form and take index_delta.  The line is drawn for each pair, not
// for its tiles, so that a new spatial order moves no pair across it.
constexpr float kNearAxis2 = 3.6e-5f, kNearAxisFar2 = 4.0e-6f, kAxisListRange2 = 2.2f;

// Pairs (slots) that the walks left to k_axis_pairs, sized for 16 an atom.  A
// count beyond the capacity says that not all of them are here; it takes 64
// bits because the pairs of a long chain do not fit an int.
struct AxisList {
    int2* pairs;
    unsigned long long* count;
    unsigned long long cap;
};

__device__ __forceinline__ void axis_push(const AxisList& A, int i, int j) {
    const unsigned long long k = atomicAdd(A.count, 1ull);
    if (k < A.cap) A.pairs[k] = make_int2(i, j);
}

// fix_add of a pair's 13 sums (I's six, J's six, the energy) on top of the
// walks', which alone the scale is sized for: a word that leaves its range
// shows by its sign.  All the adds are on their way before the first old value
// is looked at (one after the other they took 4 us more).
__device__ __forceinline__ void fix_add_checked(const FixAcc& F, int n_pad, int i, int j, const float (&v)[13]) {
    bool bad = false;
#pragma unroll
    for (int c = 0; c < 13; c++) bad |= !(fabsf(v[c]) < (float)F.limit);
    if (!bad) {
        unsigned long long a[13], old[13];
#pragma unroll
        for (int c = 0; c < 13; c++) {
            a[c] = (unsigned long long)__float2ll_rn(v[c] * (float)F.scale);
            old[c] = atomicAdd(F.acc + (size_t)(c < 12 ? c % 6 : 6) * n_pad + (c < 6 ? i : c < 12 ? j : 0), a[c]);
        }
#pragma unroll
        for (int c = 0; c < 13; c++) {
            const unsigned long long now = old[c] + a[c];
            bad |= (long long)((old[c] ^ now) & (a[c] ^ now)) < 0;
        }
    }
    if (bad) atomicExch(F.err, 1);
}

// A pair close to the x axis (slots i, j) by itself: X's azimuth is that of
// (d_y, d_z), so such a pair amplifies every rounding on the way to it by
// r / |(d_y, d_z)|.  It takes the reference's orientation (lower index first)
// and Gram-Schmidt sequence and the index-order displacement, so that its
// result depends neither on the spatial sort nor on the walk that met it.
// Both atoms' forces and torques, and the energy (word 6 n_pad), go into the
// accumulator.
__device__ __forceinline__ void axis_pair(const PairParams& P, const IndexRecords& R, const int* __restrict__ order,
                                          const double* __restrict__ pos, const FixAcc& fix, int n_pad, int i,
                                          int j) {
    const int id_i = order[i], id_j = order[j];
    const int lo = id_i < id_j ? i : j, hi = id_i < id_j ? j : i;
    float dx, dy, dz;
    index_delta(P, R, pos, lo, hi, min(id_i, id_j), max(id_i, id_j), dx, dy, dz);
    const float4 pl = R.posq_s[lo], dl = R.dipt_s[lo], ul = R.ind_s[lo];
    const float4 ph = R.posq_s[hi], dh = R.dipt_s[hi], uh = R.ind_s[hi];
    const f2 DX = bc2(dx), DY = bc2(dy), DZ = bc2(dz), R2 = dot2(DX, DY, DZ, DX, DY, DZ);
    float r2, t;
    un2(R2, r2, t);
    const f2 RINV = bc2(rsqrtf(r2));
    const f2 ZX = mul2(DX, RINV), ZY = mul2(DY, RINV), ZZ = mul2(DZ, RINV);
    const bool yz = yz_differ_slot(dy, dz, pos, lo, hi);
    f2 XX = add2(ZX, bc2(yz ? 1.0f : 0.0f)), XY = add2(ZY, bc2(yz ? 0.0f : 1.0f)), XZ = ZZ;
    const f2 NDT = neg2(dot2(ZX, ZY, ZZ, XX, XY, XZ));
    XX = fma2(ZX, NDT, XX);
    XY = fma2(ZY, NDT, XY);
    XZ = fma2(ZZ, NDT, XZ);
    float xn;
    un2(dot2(XX, XY, XZ, XX, XY, XZ), xn, t);
    const f2 SN = bc2(xn > 0.0f ? rsqrtf(xn) : 1.0f);
    XX = mul2(XX, SN);
    XY = mul2(XY, SN);
    XZ = mul2(XZ, SN);
    const QiPair o =
        qi_pair2(P, DX, DY, DZ, R2, RINV, r2, r2, XX, XY, XZ, bc2(pl.w), bc2(dl.x), bc2(dl.y), bc2(dl.z), bc2(ul.x),
                 bc2(ul.y), bc2(ul.z), dl.w, 1.0f / dl.w, bc2(ph.w), bc2(dh.x), bc2(dh.y), bc2(dh.z), bc2(uh.x),
                 bc2(uh.y), bc2(uh.z), dh.w, dh.w, 1.0f / dh.w, 1.0f / dh.w);
    const f2 I[6] = {o.nfx, o.nfy, o.nfz, xneg2(o.tx), xneg2(o.ty), xneg2(o.tz)};
    const f2 K[6] = {xneg2(o.nfx), xneg2(o.nfy), xneg2(o.nfz), xneg2(o.ux), xneg2(o.uy), xneg2(o.uz)};
    float v[13];
#pragma unroll
    for (int c = 0; c < 6; c++) {
        un2(I[c], v[c], t);
        un2(K[c], v[6 + c], t);
    }
    un2(o.e2, v[12], t);
    v[12] *= 0.5f;
    fix_add_checked(fix, n_pad, lo, hi, v);
}

// f: I side (force; sum of V, or the torque in MODE 2), g: the same for J atom
// ((lane + s1) & 15) | (lane & 16).
// MODE 3: only the pairs that the other modes leave to k_axis_pairs, evaluated
// here by axis_pair.
// OPEN: the charge-charge energy in FP64 (xi: the I atom's position, XJ: the J
// atoms'), from the FP32 1/r by one Newton step.  The energy of an open system
// is the small remainder of charge sums that grow with n^2 (20 e^2/nm of
// 1.6e6 at 3,993 atoms): in FP32 the roundings of 1/r and of the sum left
// 1e-6 to 5e-6 of it.
template <int MODE, bool FOLD, bool MASK, bool OPEN>
__device__ __forceinline__ void energy_item_walk(const PairParams& P, const double* __restrict__ pos,
                                                 const IndexRecords& R, const AxisList& axis,
                                                 const int* __restrict__ order, const FixAcc& fix, int n_pad,
                                                 const EItemTile& T, int lane, int i, int id, int jbase, float oix,
                                                 float oiy, float oiz, float4 pi, float4 di, float4 ui, unsigned mk,
                                                 unsigned fm, float damp_r2, int s0, int s1, float (&f)[6],
                                                 float (&g)[6], float& en, d3 xi, const EItemPos* XJ, double& en64) {
    const int nxt = (lane + 1) & 31;
    const f2 OX = bc2(oix), OY = bc2(oiy), OZ = bc2(oiz);
    const f2 QI = bc2(pi.w), HALF = bc2(0.5f), NTHREE = bc2(-3.0f), ONE = bc2(1.0f);
    // MODE 0: P_i in place of m_i.
    const f2 MIX = bc2(MODE == 0 ? di.x + ui.x : di.x), MIY = bc2(MODE == 0 ? di.y + ui.y : di.y),
             MIZ = bc2(MODE == 0 ? di.z + ui.z : di.z);
    const f2 UIX = bc2(ui.x), UIY = bc2(ui.y), UIZ = bc2(ui.z);
    const float ti = di.w, iti = 1.0f / di.w;
    const bool mutual = P.mutual != 0;
    f2 Lx = 0, Ly = 0, Lz = 0, Ix = 0, Iy = 0, Iz = 0, NTx = 0, NTy = 0, NTz = 0;
    if (FOLD) {
        Lx = bc2(-(float)P.box[0]);
        Ly = bc2(-(float)P.box[1]);
        Lz = bc2(-(float)P.box[2]);
        Ix = bc2((float)P.inv_box[0]);
        Iy = bc2((float)P.inv_box[1]);
        Iz = bc2((float)P.inv_box[2]);
        NTx = bc2(-(float)(P.half_box_tol[0] * P.half_box_tol[0]));
        NTy = bc2(-(float)(P.half_box_tol[1] * P.half_box_tol[1]));
        NTz = bc2(-(float)(P.half_box_tol[2] * P.half_box_tol[2]));
    }
    f2 FX = 0, FY = 0, FZ = 0, TX = 0, TY = 0, TZ = 0, EN = 0;        // I side
    f2 GX = 0, GY = 0, GZ = 0, UX = 0, UY = 0, UZ = 0;                // J side (packed atoms m, m + 16)
#pragma unroll 1
    for (int s = s0; s < s1; s++) {
        const int m = (lane + s) & 15;
        const float4 a = T.p0[m], b = T.p1[m], c = T.d0[m], d = T.d1[m], e = T.u0[m], h = T.u1[m];
        const int2 jd = T.id[m];
        f2 DX = sub2(pk2(a.x, a.y), OX), DY = sub2(pk2(a.z, a.w), OY), DZ = sub2(pk2(b.x, b.y), OZ);
        const int ja = jbase + m, jb = ja + 16;
        if (FOLD) {
            // As in xslot_pairs: one sign-bit AND of the d^2 - t^2 words flags
            // the pairs within the margin of half a box.
            f2 neg = ~0ull;
            if (fm & 1u) {
                DX = fold2(DX, Lx, Ix);
                neg &= fma2(DX, DX, NTx);
            }
            if (fm & 2u) {
                DY = fold2(DY, Ly, Iy);
                neg &= fma2(DY, DY, NTy);
            }
            if (fm & 4u) {
                DZ = fold2(DZ, Lz, Iz);
                neg &= fma2(DZ, DZ, NTz);
            }
            const f2 flag = ~neg & 0x8000000080000000ull;
            if (flag) {
                float ax, bx, ay, by, az, bz;
                un2(DX, ax, bx);
                un2(DY, ay, by);
                un2(DZ, az, bz);
                if (((flag >> 31) & 1ull) && i < P.n && ja < P.n) {
                    const d3 q = exact_delta(P, pos, i, ja);
                    ax = (float)q.x;
                    ay = (float)q.y;
                    az = (float)q.z;
                }
                if ((flag >> 63) && i < P.n && jb < P.n) {
                    const d3 q = exact_delta(P, pos, i, jb);
                    bx = (float)q.x;
                    by = (float)q.y;
                    bz = (float)q.z;
                }
                DX = pk2(ax, bx);
                DY = pk2(ay, by);
                DZ = pk2(az, bz);
            }
        }
        // Orientation: sign bits set where the I atom has the higher index.
        const f2 SG = pk2(__int_as_float((jd.x - id) & 0x80000000), __int_as_float((jd.y - id) & 0x80000000));
        const f2 QJS = pk2(b.z, b.w) ^ SG, QIS = QI ^ SG;
        const f2 MJX = pk2(c.x, c.y), MJY = pk2(c.z, c.w), MJZ = pk2(d.x, d.y);
        const f2 UJX = pk2(e.x, e.y), UJY = pk2(e.z, e.w), UJZ = pk2(h.x, h.y);
        const f2 RHO2 = fma2(DY, DY, mul2(DZ, DZ));
        const f2 R2 = fma2(DX, DX, RHO2);
        float r2a, r2b, ra, rb;
        un2(R2, r2a, r2b);
        un2(RHO2, ra, rb);
        if (MASK) {
            r2a = (mk >> m) & 1u ? r2a : INFINITY;
            r2b = (mk >> (m + 16)) & 1u ? r2b : INFINITY;
        }
        f2 RINV = pk2(rsqrtf(r2a), rsqrtf(r2b));
        // Frame X row.
        const f2 XS = mul2(RINV, pk2(rsqrtf(ra), rsqrtf(rb)));
        const f2 NDXS = mul2(xneg2(DX), XS);
        f2 XX = mul2(RHO2, XS), XY = mul2(NDXS, DY), XZ = mul2(NDXS, DZ);
        if (ra <= kNearAxis2 || rb <= kNearAxis2) {
            float xr[2], rv[2], xx[2], xy[2], xz[2], dx[2], dy[2], dz[2];
            un2(DX, dx[0], dx[1]);
            un2(DY, dy[0], dy[1]);
            un2(DZ, dz[0], dz[1]);
            un2(RINV, rv[0], rv[1]);
            un2(XX, xx[0], xx[1]);
            un2(XY, xy[0], xy[1]);
            un2(XZ, xz[0], xz[1]);
            xr[0] = ra;
            xr[1] = rb;
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int j = k ? jb : ja;
                float& r2 = k ? r2b : r2a;
                const bool listed = MODE == 2 || (MODE == 3 && !P.lab_energy) || r2 < kAxisListRange2 * P.damp_r2;
                if (xr[k] > (listed ? kNearAxis2 : kNearAxisFar2)) continue;
                if (MODE == 3) {
                    if (listed && r2 < INFINITY) axis_pair(P, R, order, pos, fix, n_pad, i, j);
                    continue;
                }
                if (listed) {
                    if (r2 < INFINITY) {
                        axis_push(axis, i, j);
                        r2 = INFINITY;
                        rv[k] = 0.0f;
                    }
                } else if (r2 < INFINITY) {
                    index_delta(P, R, pos, i, j, id, k ? jd.y : jd.x, dx[k], dy[k], dz[k]);
                    const float h2 = fmaf(dy[k], dy[k], dz[k] * dz[k]);
                    rv[k] = rsqrtf(fmaf(dx[k], dx[k], h2));
                    const float s = rv[k] * rsqrtf(h2);
                    xx[k] = h2 * s;
                    xy[k] = -dx[k] * s * dy[k];
                    xz[k] = -dx[k] * s * dz[k];
                    xr[k] = h2;
                }
                if (xr[k] <= 1.0e-10f)
                    qi_frame_x(dx[k], dy[k], dz[k], rv[k], yz_differ_slot(dy[k], dz[k], pos, i, j), xx[k], xy[k],
                               xz[k]);
            }
            RINV = pk2(rv[0], rv[1]);
            XX = pk2(xx[0], xx[1]);
            XY = pk2(xy[0], xy[1]);
            XZ = pk2(xz[0], xz[1]);
        }
        if constexpr (MODE == 3) continue;
        if constexpr (MODE == 2) {
            const QiPair o = qi_pair2(P, DX, DY, DZ, R2, RINV, r2a, r2b, XX, XY, XZ, QIS, MIX, MIY, MIZ, UIX, UIY, UIZ,
                                      ti, iti, QJS, MJX, MJY, MJZ, UJX, UJY, UJZ, d.z, d.w, h.z, h.w);
            const f2 SFX = o.nfx ^ SG, SFY = o.nfy ^ SG, SFZ = o.nfz ^ SG;
            FX = add2(FX, SFX);
            FY = add2(FY, SFY);
            FZ = add2(FZ, SFZ);
            GX = sub2(GX, SFX);
            GY = sub2(GY, SFY);
            GZ = sub2(GZ, SFZ);
            TX = sub2(TX, o.tx);
            TY = sub2(TY, o.ty);
            TZ = sub2(TZ, o.tz);
            UX = sub2(UX, o.ux);
            UY = sub2(UY, o.uy);
            UZ = sub2(UZ, o.uz);
            EN = fma2(HALF, o.e2, EN);
        } else {
            const f2 MI0 = dot2(XX, XY, XZ, MIX, MIY, MIZ), UI0 = dot2(XX, XY, XZ, UIX, UIY, UIZ);
            const f2 MJ0 = dot2(XX, XY, XZ, MJX, MJY, MJZ), UJ0 = dot2(XX, XY, XZ, UJX, UJY, UJZ);
            const f2 rv2 = mul2(RINV, RINV), rv3 = mul2(rv2, RINV);
            const f2 NR3 = mul2(NTHREE, rv3), R3T = add2(rv3, rv3);
            const f2 qq = mul2(QIS, QJS);
            const f2 RQJ = mul2(rv2, QJS), RQI = mul2(rv2, xneg2(QIS));
            f2 KX, KY, KZ, QF, RAD;   // K, radial force term, 2 r^2 (E without q_i q_j/r and the V terms)
            if constexpr (MODE == 0) {
                RAD = fma2(QJS, MI0, mul2(xneg2(QIS), MJ0));
                const f2 A = fma2(NR3, MJ0, RQJ), B = fma2(NR3, MI0, RQI);
                TX = fma2(A, XX, fma2(rv3, MJX, TX));
                TY = fma2(A, XY, fma2(rv3, MJY, TY));
                TZ = fma2(A, XZ, fma2(rv3, MJZ, TZ));
                UX = fma2(B, XX, fma2(rv3, MIX, UX));
                UY = fma2(B, XY, fma2(rv3, MIY, UY));
                UZ = fma2(B, XZ, fma2(rv3, MIZ, UZ));
                const f2 NRK = mutual ? NR3 : xneg2(NR3);
                const f2 CI = mul2(NRK, UJ0), CJ = mul2(NRK, UI0);
                KX = fma2(A, MIX, fma2(B, MJX, fma2(CI, UIX, mul2(CJ, UJX))));
                KY = fma2(A, MIY, fma2(B, MJY, fma2(CI, UIY, mul2(CJ, UJY))));
                KZ = fma2(A, MIZ, fma2(B, MJZ, fma2(CI, UIZ, mul2(CJ, UJZ))));
                QF = fma2(R3T, RAD, mul2(rv2, qq));
            } else {
                // Thole factors (1 beyond damp_r2 or where t_i t_j <= 1e-5, as the reference).
                f2 TC = ONE, W = ONE, T0 = ONE;
                if (r2a < damp_r2 || r2b < damp_r2) {
                    const f2 U = mul2(mul2(mul2(R2, RINV), bc2(iti)), pk2(h.z, h.w));
                    const f2 AU3 = mul2(pk2(fminf(ti, d.z), fminf(ti, d.w)), mul2(U, mul2(U, U)));
                    float xa, xb;
                    un2(AU3, xa, xb);
                    const bool da = r2a < damp_r2 && fabsf(ti * d.z) > 1.0e-5f;
                    const bool db = r2b < damp_r2 && fabsf(ti * d.w) > 1.0e-5f;
                    const f2 NEX = pk2(da ? -__expf(-xa) : 0.0f, db ? -__expf(-xb) : 0.0f);
                    const f2 X3 = pk2(da ? xa : 0.0f, db ? xb : 0.0f);   // no inf/NaN into the products
                    TC = add2(ONE, NEX);
                    W = fma2(NEX, add2(X3, ONE), ONE);
                    T0 = fma2(NEX, fma2(bc2(1.5f), X3, ONE), ONE);
                }
                const f2 CM = fma2(QJS, MI0, mul2(xneg2(QIS), MJ0)), CU = fma2(QJS, UI0, mul2(xneg2(QIS), UJ0));
                RAD = fma2(TC, CU, CM);
                const f2 A = fma2(NR3, fma2(W, UJ0, MJ0), RQJ), B = fma2(NR3, fma2(W, UI0, MI0), RQI);
                const f2 R3C = mul2(rv3, TC);
                TX = fma2(A, XX, fma2(rv3, MJX, fma2(R3C, UJX, TX)));
                TY = fma2(A, XY, fma2(rv3, MJY, fma2(R3C, UJY, TY)));
                TZ = fma2(A, XZ, fma2(rv3, MJZ, fma2(R3C, UJZ, TZ)));
                UX = fma2(B, XX, fma2(rv3, MIX, fma2(R3C, UIX, UX)));
                UY = fma2(B, XY, fma2(rv3, MIY, fma2(R3C, UIY, UY)));
                UZ = fma2(B, XZ, fma2(rv3, MIZ, fma2(R3C, UIZ, UZ)));
                const f2 LAM = bc2(mutual ? 2.0f : 0.0f), NRW = mul2(NR3, W);
                const f2 CI = fma2(NRW, fma2(LAM, UJ0, MJ0), mul2(TC, RQJ));
                const f2 CJ = fma2(NRW, fma2(LAM, UI0, MI0), mul2(TC, RQI));
                KX = fma2(A, MIX, fma2(B, MJX, fma2(CI, UIX, mul2(CJ, UJX))));
                KY = fma2(A, MIY, fma2(B, MJY, fma2(CI, UIY, mul2(CJ, UJY))));
                KZ = fma2(A, MIZ, fma2(B, MJZ, fma2(CI, UIZ, mul2(CJ, UJZ))));
                QF = fma2(R3T, fma2(T0, CU, CM), mul2(rv2, qq));
            }
            if constexpr (OPEN) {
                EN = fma2(mul2(HALF, rv2), RAD, EN);
                float rva, rvb;
                un2(RINV, rva, rvb);
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const int jj = m + 16 * k;
                    const double x = XJ->x[jj] - xi.x, y = XJ->y[jj] - xi.y, z = XJ->z[jj] - xi.z;
                    const double r2 = x * x + y * y + z * z, y0 = (double)(k ? rvb : rva);
                    const double r1 = y0 + (0.5 * y0) * (1.0 - (r2 * y0) * y0);
                    en64 += ((double)pi.w * (double)(k ? b.w : b.z)) * r1;
                }
            } else {
                EN = fma2(RINV, qq, fma2(mul2(HALF, rv2), RAD, EN));
            }
            // f = (rinv K.X + QF) X - rinv K, with the orientation's sign.
            const f2 CF = fma2(RINV, dot2(KX, KY, KZ, XX, XY, XZ), QF) ^ SG;
            const f2 NR = xneg2(RINV) ^ SG;
            const f2 FVX = fma2(CF, XX, mul2(NR, KX)), FVY = fma2(CF, XY, mul2(NR, KY)),
                     FVZ = fma2(CF, XZ, mul2(NR, KZ));
            FX = sub2(FX, FVY);
            FY = sub2(FY, FVZ);
            FZ = sub2(FZ, FVX);
            GX = add2(GX, FVY);
            GY = add2(GY, FVZ);
            GZ = add2(GZ, FVX);
        }
        GX = __shfl_sync(kFull, GX, nxt);
        GY = __shfl_sync(kFull, GY, nxt);
        GZ = __shfl_sync(kFull, GZ, nxt);
        UX = __shfl_sync(kFull, UX, nxt);
        UY = __shfl_sync(kFull, UY, nxt);
        UZ = __shfl_sync(kFull, UZ, nxt);
    }
    float lo, hi;
    const f2 Is[6] = {FX, FY, FZ, TX, TY, TZ}, Js[6] = {GX, GY, GZ, UX, UY, UZ};
#pragma unroll
    for (int k = 0; k < 6; k++) {
        un2(Is[k], lo, hi);
        f[k] = lo + hi;
        // Lanes l and l ^ 16 hold the two copies of atoms (m, m + 16).
        un2(Js[k], lo, hi);
        const float olo = __shfl_xor_sync(kFull, lo, 16), ohi = __shfl_xor_sync(kFull, hi, 16);
        g[k] = lane < 16 ? lo + olo : hi + ohi;
    }
    un2(EN, lo, hi);
    en = lo + hi;
}

// Sum of V -> torque -perm(m x V) and the dipole energy 0.5 m.V (MODE 0, 1).
__device__ __forceinline__ float torque_of_v(float4 m, float (&f)[6]) {
    const float vx = f[3], vy = f[4], vz = f[5];
    f[3] = -(m.z * vx - m.x * vz);
    f[4] = -(m.x * vy - m.y * vx);
    f[5] = -(m.y * vz - m.z * vy);
    return 0.5f * (m.x * vx + m.y * vy + m.z * vz);
}

__device__ __forceinline__ void copy16_async(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

// The J records of an item's next tile, fetched while the current one is walked.
struct EItemRaw {
    float4 p[32], d[32], u[32];
};

// Shared memory of an item.
struct EItemShared {
    EItemTile T;
    EItemRaw raw;
    double my[6][32];
};

// Records and tables of the energy items, by slot.
struct EItemArrays {
    const float4 *posq, *dipt, *indv;
    const int* order;
    const double4 *tctr, *text;
    const double* pos;
    const int *exc_off, *exc_j;
    const double *exc_m, *exc_s;
    const int2* exc_tiles;
    IndexRecords R;
    AxisList axis;
    FixAcc fix;
    int L, n_pad;
};

// Part `part` of `parts` of item `bx`: see k_energy_items.  SCAN: nothing but the
// pairs that belong to k_axis_pairs (MODE 3).
template <bool GENERAL, bool OPEN, bool SCAN>
__device__ __forceinline__ void energy_item(const PairParams& P, const EItemArrays& A, EItemShared& S, EItemPos* XJ,
                                            unsigned bx, unsigned part, unsigned parts,
                                            double* __restrict__ item_energy) {
    const int lane = threadIdx.x, L = A.L, n_pad = A.n_pad;
    const float4 *__restrict__ posq = A.posq, *__restrict__ dipt = A.dipt, *__restrict__ indv = A.indv;
    const int *__restrict__ order = A.order, *__restrict__ exc_j = A.exc_j;
    const double *__restrict__ pos = A.pos, *__restrict__ exc_m = A.exc_m, *__restrict__ exc_s = A.exc_s;
    const double4 *__restrict__ tctr = A.tctr, *__restrict__ text = A.text;
    const FixAcc& fix = A.fix;
    EItemTile& T = S.T;
    EItemRaw& raw = S.raw;
    int p, q;
    band_pair(bx / L, p, q);
    const int I = p * L + (int)(bx % L), J0 = q * L, J1 = min(J0 + L, P.n_tiles);
    int J = max(J0, I);
    if (I >= P.n_tiles || J >= J1) {
        if (!SCAN && lane == 0) *item_energy = 0.0;
        return;
    }
    const int s0 = 16 * part / parts, s1 = 16 * (part + 1) / parts;
    const float damp_r2 = kDampRange32 * P.damp_r2;
    const auto fetch = [&](int t) {
        copy16_async(&raw.p[lane], posq + t * 32 + lane);
        copy16_async(&raw.d[lane], dipt + t * 32 + lane);
        copy16_async(&raw.u[lane], indv + t * 32 + lane);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(J);
    const int i = I * 32 + lane;
    const float4 pi = posq[i], di = dipt[i], ui = indv[i];
    const int id = order[i];
    d3 xi = {0.0, 0.0, 0.0};
    if (OPEN) xi = ld3(pos + 3 * (size_t)i);
    const int2 et = A.exc_tiles[I];
    int e0 = 0, e1 = 0;
    unsigned own = 0u;
    if (i < P.n) {
        own = ~0u;
        e0 = A.exc_off[i];
        e1 = A.exc_off[i + 1];
    }
    float gdx = 0.f, gdy = 0.f, gdz = 0.f;
    unsigned gfl = 0u;
    if (lane < L && J0 + lane < P.n_tiles) {
        const TileGeom g = tile_geom(P, (double)damp_r2, tctr[I], text[I], tctr[J0 + lane], text[J0 + lane]);
        gdx = (float)g.dcx;
        gdy = (float)g.dcy;
        gdz = (float)g.dcz;
        gfl = g.fmask | (g.fold ? 8u : 0u) | (g.near ? 16u : 0u);
    }
#pragma unroll
    for (int k = 0; k < 6; k++) S.my[k][lane] = 0.0;
    double energy = 0.0;
    for (; J < J1; J++) {
        const int jbase = J * 32, jid = order[jbase + lane];
        const float dx = __shfl_sync(kFull, gdx, J - J0), dy = __shfl_sync(kFull, gdy, J - J0),
                    dz = __shfl_sync(kFull, gdz, J - J0);
        const unsigned fl = __shfl_sync(kFull, gfl, J - J0);
        unsigned mk = own;
        if (J == P.n_tiles - 1 && (P.n & 31)) mk &= (1u << (P.n & 31)) - 1u;
        if (I == J) mk &= ~((2u << lane) - 1u);   // each pair of a diagonal tile once: j > i
        if (J >= et.x && J <= et.y)
            for (int e = e0; e < e1; e++) {
                const unsigned off = (unsigned)(exc_j[e] - jbase);
                if (off < 32u && (exc_m[e] != 1.0 || exc_s[e] != 1.0)) mk &= ~(1u << off);
            }
        const bool masked = __any_sync(kFull, mk != ~0u);
        const bool plain = !GENERAL && !masked && !(fl & 16u);   // MODE 0
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        {
            const float4 pj = raw.p[lane], uj = raw.u[lane];
            float4 dj = raw.d[lane];
            if (plain) {
                dj.x += uj.x;
                dj.y += uj.y;
                dj.z += uj.z;
            }
            stage_eitem(T, lane, pj, dj, uj, jid);
            if (OPEN) {
                const d3 x = ld3(pos + 3 * (size_t)(jbase + lane));
                XJ->x[lane] = x.x;
                XJ->y[lane] = x.y;
                XJ->z[lane] = x.z;
            }
        }
        __syncwarp();
        if (J + 1 < J1) fetch(J + 1);
        const float ox = pi.x - dx, oy = pi.y - dy, oz = pi.z - dz;
        float f[6], g[6], en;
#define TDP_EWALK(M, F, K) \
    energy_item_walk<M, F, K, OPEN>(P, pos, A.R, A.axis, order, fix, n_pad, T, lane, i, id, jbase, ox, oy, oz, pi, di, \
                                    ui, mk, fl, damp_r2, s0, s1, f, g, en, xi, XJ, energy)
        if constexpr (SCAN) {
            TDP_EWALK(3, true, true);
            continue;
        } else if constexpr (GENERAL) {
            TDP_EWALK(2, true, true);
        } else if (plain) {
            if (fl & 8u) TDP_EWALK(0, true, false);
            else TDP_EWALK(0, false, false);
        } else if (masked) {
            TDP_EWALK(1, true, true);
        } else if (fl & 8u) {
            TDP_EWALK(1, true, false);
        } else {
            TDP_EWALK(1, false, false);
        }
#undef TDP_EWALK
        const int jl = ((lane + s1) & 15) | (lane & 16);
        if constexpr (!GENERAL) en += torque_of_v(di, f) + torque_of_v(dipt[jbase + jl], g);
        energy += (double)en;
#pragma unroll
        for (int k = 0; k < 6; k++) {
            fix_add(fix, (size_t)k * n_pad + jbase + jl, g[k]);
            S.my[k][lane] += (double)f[k];
        }
    }
    if constexpr (!SCAN) {
#pragma unroll
        for (int k = 0; k < 6; k++) fix_add(fix, (size_t)k * n_pad + i, S.my[k][lane]);
        energy = warp_sum(energy);
        if (lane == 0) *item_energy = energy;
    }
}

// Mixed-form energy kernel: warp items as in k_field_items, one I tile against
// J tiles [c L, c L + L), in the spatial order of the field kernels (compact
// tiles: few tile pairs fold or reach the damping range, and the FP32 offsets
// are short).  Pairs that do not count (self, padding, the second visit on a
// diagonal tile, listed partners) are masked out; k_energy_items_done
// evaluates the partners.  GENERAL: MODE 2 for every tile pair.  OPEN: no
// box, the charge energy in FP64.
//
// Bound by the FP32 pipe (82 FMA-pipe f32x2 instructions a step of two pairs
// in MODE 0, about 100 in MODE 1).  The band-pair kernel before it ran in
// index order: its tiles were as long as the input's rows (3.3 nm on a
// lattice), so most tile pairs folded, and those within the damping range
// took the quasi-internal frame walk (about 230).  Before -> now (the done
// kernels included): 31 -> 27 us at 648 atoms, 210 -> 83 at 3,993, 535 -> 409
// at 12,288, 24,200 -> 20,300 at 98,304.
template <bool GENERAL, bool OPEN>
__global__ void __launch_bounds__(32, 12)
    k_energy_items(PairParams P, EItemArrays A, double* __restrict__ energy_partial) {
    __shared__ EItemShared S;
    __shared__ EItemPos XJ;
    energy_item<GENERAL, OPEN, false>(P, A, S, &XJ, blockIdx.x, blockIdx.y, gridDim.y,
                                      energy_partial + (size_t)blockIdx.y * gridDim.x + blockIdx.x);
}

// The pairs that the walks left out, each by axis_pair: from the list, or,
// where that could not hold them, from a second pass over the items, which
// meets the same pairs.  The sums are integers, so the two give the same bits.
__global__ void __launch_bounds__(32) k_axis_pairs(PairParams P, EItemArrays A, int items) {
    __shared__ EItemShared S;
    const unsigned long long count = *A.axis.count;
    if (count <= A.axis.cap) {
        for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < (int)count; q += gridDim.x * blockDim.x) {
            const int2 ij = A.axis.pairs[q];
            axis_pair(P, A.R, A.order, A.pos, A.fix, A.n_pad, ij.x, ij.y);
        }
        return;
    }
    for (int bx = blockIdx.x; bx < items; bx += gridDim.x)
        energy_item<false, false, true>(P, A, S, nullptr, bx, 0, 1, nullptr);
}

// Fixed-point force and torque sums -> FP64 in index order, clearing them,
// plus each slot's listed partners one-sided with their scales (FP64 pair
// routine on the pair records; the pair's energy counts on its lower index),
// and the block's share of the item energies, summed in order into
// energy_block[blockIdx.x].
__global__ void k_energy_items_done(PairParams P, const float4* __restrict__ posq, const float4* __restrict__ dipt,
                                    const float4* __restrict__ indv, const int* __restrict__ order,
                                    const double* __restrict__ pos, const int* __restrict__ exc_off,
                                    const int* __restrict__ exc_j, const double* __restrict__ exc_m,
                                    const double* __restrict__ exc_s, IndexRecords R,
                                    unsigned long long* __restrict__ axis_count,
                                    int n_pad, unsigned long long* __restrict__ acc, double inv_scale, int n_items,
                                    const double* __restrict__ energy_item, double* __restrict__ fpair,
                                    double* __restrict__ torque, double* __restrict__ energy_block) {
    __shared__ double red[40];
    const int per = (n_items + gridDim.x - 1) / gridDim.x;
    const int a0 = min(n_items, blockIdx.x * per), a1 = min(n_items, a0 + per);
    double energy = 0.0;
    for (int a = a0 + threadIdx.x; a < a1; a += blockDim.x) energy += energy_item[a];
    if (blockIdx.x == 0 && threadIdx.x == 0) {   // the listed pairs' energy; the list is empty again
        energy += (double)(long long)acc[6 * (size_t)n_pad] * inv_scale;
        acc[6 * (size_t)n_pad] = 0ull;
        *axis_count = 0ull;
    }
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n_pad) {
        double v[6];
#pragma unroll
        for (int c = 0; c < 6; c++) {
            v[c] = (double)(long long)acc[(size_t)c * n_pad + k] * inv_scale;
            acc[(size_t)c * n_pad + k] = 0ull;
        }
        if (k < P.n) {
            const int id = order[k];
            const double4 p = make_double4(0, 0, 0, posq[k].w);
            const float4 df = dipt[k], uf = indv[k];
            const EAtom<double> me = eatom<double>(p, make_double4(df.x, df.y, df.z, df.w),
                                                   make_double4(uf.x, uf.y, uf.z, 0));
            for (int e = exc_off[k]; e < exc_off[k + 1]; e++) {
                const double mS = exc_m[e], iS = exc_s[e];
                if ((mS == 0.0 && iS == 0.0) || (mS == 1.0 && iS == 1.0)) continue;
                const int j = exc_j[e];
                const float4 dj = dipt[j], uj = indv[j];
                const EAtom<double> other = eatom<double>(make_double4(0, 0, 0, posq[j].w),
                                                          make_double4(dj.x, dj.y, dj.z, dj.w),
                                                          make_double4(uj.x, uj.y, uj.z, 0));
                float dx, dy, dz;
                index_delta(P, R, pos, k, j, id, order[j], dx, dy, dz);
                const d3 d = {(double)dx, (double)dy, (double)dz};
                const double r2 = dot(d, d);
                const bool yzd = pos[3 * (size_t)k + 1] != pos[3 * (size_t)j + 1] ||
                                 pos[3 * (size_t)k + 2] != pos[3 * (size_t)j + 2];
                const double dr2 = (double)P.damp_r2, p4 = P.rinv4_power, f4 = P.rinv4_fill;
                if (id < order[j])
                    pair_energy<double, true>(d.x, d.y, d.z, r2, yzd, me, other, mS, iS, dr2, p4, f4, P.mutual != 0,
                                              v[0], v[1], v[2], v[3], v[4], v[5], energy);
                else
                    pair_energy<double, false>(-d.x, -d.y, -d.z, r2, yzd, other, me, mS, iS, dr2, p4, f4,
                                               P.mutual != 0, v[0], v[1], v[2], v[3], v[4], v[5], energy);
            }
#pragma unroll
            for (int c = 0; c < 3; c++) {
                fpair[3 * (size_t)id + c] = v[c];
                torque[3 * (size_t)id + c] = v[3 + c];
            }
        }
    }
    energy = block_sum(energy, red);
    if (threadIdx.x == 0) energy_block[blockIdx.x] = energy;
}

// Partner pairs of a SLOW tile pair with their (M, I) scales, each side once:
// the lane's I atom with its partners in J (the pair energy is counted on the
// lower-index side), and atom l of J (off the diagonal) with its partners in I.
template <bool FOLD>
__device__ __forceinline__ void energy_partners(
    const PairParams& P, const double2* __restrict__ yz, const double4* __restrict__ posq,
    const double4* __restrict__ dipt, const double4* __restrict__ indv, const ERec64& T, int j0,
    const int* __restrict__ exc_off, const int* __restrict__ exc_j, const double* __restrict__ exc_m,
    const double* __restrict__ exc_s, const TileGeom& geo, double4 cA, double4 cB, int lane, int i, int ibase,
    int jbase, int e0, int e1, double oix, double oiy, double oiz, const EAtom<double>& me, bool diag, double f[6],
    double g[6], double& en) {
    const int nmax = P.n_tiles * 32 - 1;
    const double damp_r2 = (double)P.damp_r2, rv4p = (double)P.rinv4_power, rv4f = (double)P.rinv4_fill;
#pragma unroll 1
    for (int e = e0; e < e1; e++) {
        unsigned off = (unsigned)(exc_j[e] - jbase);
        if (off >= 32u) continue;
        const double mS = exc_m[e], iS = exc_s[e];
        if (mS == 0.0 && iS == 0.0) continue;
        const int j = jbase + (int)off, k = j0 + (int)off;
        const EAtom<double> other = T.atom(k);
        double dx, dy, dz;
        pair_delta<FOLD>(P, geo.fmask, T.xy[k].x, T.xy[k].y, T.zq[k].x, oix, oiy, oiz, dx, dy, dz);
        const double r2 = dx * dx + dy * dy + dz * dz;
        const bool yzd = yz_differ<double>(dy, dz, yz, i, j, nmax);
        if (j > i)
            pair_energy<double, true>(dx, dy, dz, r2, yzd, me, other, mS, iS, damp_r2, rv4p, rv4f, P.mutual != 0, f[0],
                                      f[1], f[2], f[3], f[4], f[5], en);
        else
            pair_energy<double, false>(-dx, -dy, -dz, r2, yzd, other, me, mS, iS, damp_r2, rv4p, rv4f, P.mutual != 0,
                                       f[0], f[1], f[2], f[3], f[4], f[5], en);
    }
    if (diag) return;
    const int jl = jbase + lane, kl = j0 + lane;
    if (jl >= P.n) return;
    const EAtom<double> mine = T.atom(kl);
    double dummy = 0;
#pragma unroll 1
    for (int e = exc_off[jl]; e < exc_off[jl + 1]; e++) {
        const int a = exc_j[e];
        if ((unsigned)(a - ibase) >= 32u) continue;
        const double mS = exc_m[e], iS = exc_s[e];
        if (mS == 0.0 && iS == 0.0) continue;
        const double4 pa = posq[a];
        const EAtom<double> A = eatom<double>(pa, dipt[a], indv[a]);
        double ox, oy, oz;
        shift_into(geo, cA, cB, pa.x, pa.y, pa.z, ox, oy, oz);
        double dx, dy, dz;  // p_jl - p_a: a (tile I < J) is the lower index
        pair_delta<FOLD>(P, geo.fmask, T.xy[kl].x, T.xy[kl].y, T.zq[kl].x, ox, oy, oz, dx, dy, dz);
        const double r2 = dx * dx + dy * dy + dz * dz;
        const bool yzd = yz_differ<double>(dy, dz, yz, a, jl, nmax);
        pair_energy<double, false>(dx, dy, dz, r2, yzd, A, mine, mS, iS, damp_r2, rv4p, rv4f, P.mutual != 0, g[0],
                                   g[1], g[2], g[3], g[4], g[5], dummy);
    }
}

// Plain form: one CTA per band pair, one warp per I tile at a time (one to four
// warps).  Bound by the FP64 chain (135 operations a pair, the pipe 54 % busy
// with 12 warps an SM).  Warps without a tile in narrow bands are not launched,
// the records lie in conflict-free pieces, and the pairs beyond the damping
// range take pair_energy_lab: 81 -> 59 us at 1,029 atoms, 427 -> 220 at 3,993,
// 1205 -> 1130 at 12,288.
__global__ void __launch_bounds__(kSymThreads, 3) k_energy_sym(
    PairParams P, const double4* __restrict__ posq, const double4* __restrict__ dipt,
    const double4* __restrict__ indv, const double2* __restrict__ yz, const double4* __restrict__ tctr,
    const double4* __restrict__ text, const double* __restrict__ pos, const int* __restrict__ exc_off,
    const int* __restrict__ exc_j, const double* __restrict__ exc_m, const double* __restrict__ exc_s,
    const int2* __restrict__ exc_tiles, int n_pad, double* __restrict__ partial, double* __restrict__ energy_partial) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int BT = P.band_tiles, NA = BT * 32;
    double* s_acc = reinterpret_cast<double*>(smem);              // 6 * NA: J-side sums of band q
    double* s_iacc = s_acc + 6 * NA;                               // 7 * threads: I-side sums and energy
    double4* s_ctr = reinterpret_cast<double4*>(s_iacc + 7 * blockDim.x);
    double4* s_ext = s_ctr + BT;
    const ERec64 T(reinterpret_cast<double2*>(s_ext + BT), NA);

    int p, q;
    band_pair(blockIdx.x, p, q);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int qa0 = q * NA;
    for (int k = threadIdx.x; k < NA; k += blockDim.x) {
        const double4 a = posq[qa0 + k], b = dipt[qa0 + k], u = indv[qa0 + k];
        T.xy[k] = make_double2(a.x, a.y);
        T.zq[k] = make_double2(a.z, a.w);
        T.mm[k] = make_double2(b.x, b.y);
        T.mu[k] = make_double2(b.z, u.x);
        T.uu[k] = make_double2(u.y, u.z);
        T.t[k] = b.w;
        for (int c = 0; c < 6; c++) s_acc[c * NA + k] = 0.0;
    }
    for (int k = threadIdx.x; k < BT; k += blockDim.x) {
        s_ctr[k] = tctr[q * BT + k];
        s_ext[k] = text[q * BT + k];
    }
    double* my = s_iacc + 7 * threadIdx.x;
    my[6] = 0.0;
    __syncthreads();

    const int stride = BT / warps;
    const int rounds = (BT + warps - 1) / warps;
    for (int r = 0; r < rounds; r++) {
        const int Il = warp + warps * r;
        const int I = p * BT + Il;
        const bool wact = Il < BT && I < P.n_tiles;
        const int ibase = I * 32;
        const int i = ibase + lane;
        double4 pi = {}, di = {}, ui = {};
        double4 cA = {}, eA = {};
        int2 et = make_int2(1 << 30, -1);
        int e0 = 0, e1 = 0;
        if (wact) {
            pi = posq[i];
            di = dipt[i];
            ui = indv[i];
            cA = tctr[I];
            eA = text[I];
            et = exc_tiles[I];
            if (i < P.n) {
                e0 = exc_off[i];
                e1 = exc_off[i + 1];
            }
        }
        const EAtom<double> me = eatom<double>(pi, di, ui);
        for (int c = 0; c < 6; c++) my[c] = 0.0;
        for (int t = 0; t < BT; t++) {
            const int Jl = (t + warp * stride) % BT;
            const int J = q * BT + Jl;
            if (wact && J < P.n_tiles && (p != q || Jl >= Il)) {
                const double4 cB = s_ctr[Jl];
                const bool diag = I == J;
                const bool slow = diag || (J == P.n_tiles - 1 && (P.n & 31)) || (J >= et.x && J <= et.y);
                const TileGeom g = tile_geom(P, (double)P.damp_r2, cA, eA, cB, s_ext[Jl]);
                double oix, oiy, oiz;
                shift_into(g, cA, cB, pi.x, pi.y, pi.z, oix, oiy, oiz);
                const int jbase = J * 32, j0 = Jl * 32;
                const unsigned partners = slow ? partner_bits(exc_j, e0, e1, jbase) : 0u;
                double f[6] = {0, 0, 0, 0, 0, 0}, gg[6] = {0, 0, 0, 0, 0, 0}, en = 0;
#define TDP_EWALK64(F, S, L) \
    energy_walk<F, S, L>(P, yz, T, j0, lane, i, jbase, oix, oiy, oiz, me, diag, partners, g.fmask, f, gg, en)
#define TDP_EPARTNERS64(F)                                                                                       \
    energy_partners<F>(P, yz, posq, dipt, indv, T, j0, exc_off, exc_j, exc_m, exc_s, g, cA, cB, lane, i, ibase, \
                       jbase, e0, e1, oix, oiy, oiz, me, diag, f, gg, en)
                if (slow) {
                    if (g.fold) {
                        TDP_EWALK64(true, true, false);
                        TDP_EPARTNERS64(true);
                    } else {
                        TDP_EWALK64(false, true, false);
                        TDP_EPARTNERS64(false);
                    }
                } else if (!g.near && P.lab_energy) {
                    if (g.fold) TDP_EWALK64(true, false, true);
                    else TDP_EWALK64(false, false, true);
                } else if (g.fold) {
                    TDP_EWALK64(true, false, false);
                } else {
                    TDP_EWALK64(false, false, false);
                }
#undef TDP_EWALK64
#undef TDP_EPARTNERS64
                double* acc = s_acc + Jl * 32 + lane;
                for (int c = 0; c < 6; c++) {
                    acc[c * NA] += gg[c];
                    my[c] += f[c];
                }
                my[6] += en;
            }
            // Within a window of `stride` steps the warps' J tiles are
            // disjoint ((t + warp * stride) % BT), so the shared J-side sums
            // need a barrier only between windows; the windows' order fixes the
            // order of the additions (deterministic).
            if ((t + 1) % stride == 0 || t + 1 == BT) __syncthreads();
        }
        if (wact) {
            if (p == q) {
                double* acc = s_acc + Il * 32 + lane;
                for (int c = 0; c < 6; c++) acc[c * NA] += my[c];
            } else {
                const size_t b = (size_t)q * 6 * n_pad;
                for (int c = 0; c < 6; c++) partial[b + (size_t)c * n_pad + i] = my[c];
            }
        }
        __syncthreads();
    }
    const size_t b = (size_t)p * 6 * n_pad;
    for (int k = threadIdx.x; k < NA; k += blockDim.x)
        for (int c = 0; c < 6; c++) partial[b + (size_t)c * n_pad + qa0 + k] = s_acc[c * NA + k];
    // CTA energy, summed in thread order (padding atoms contribute exactly 0).
    double e = warp_sum(my[6]);
    __shared__ double s_red[kSymWarps];
    if (lane == 0) s_red[warp] = e;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < warps; w++) s += s_red[w];
        energy_partial[blockIdx.x] = s;
    }
}

size_t field_smem(int BT) {
    return (size_t)32 * BT * (4 * sizeof(double2) + (1 + 3 * (BT / 2)) * sizeof(double)) + BT * BT * sizeof(double4);
}

size_t energy_smem(int BT) {
    const int NA = 32 * BT;
    return sizeof(double) * (7 * NA + 7 * kSymThreads) + sizeof(double4) * 2 * BT + sizeof(double2) * 5 * NA;
}

int band_pairs(const Dev& d) { return d.pp.n_bands * (d.pp.n_bands + 1) / 2; }

FixAcc fix_of(const Dev& d) { return FixAcc{d.fixacc, d.fix_err, d.fix_scale, d.fix_limit}; }

// Plain form: the slots of every sum, in slot order, into slot 0, one thread
// per sum.  The consumers used to add an atom's slots themselves, 3 x n_bands
// dependent loads on one thread an atom: at 12,288 atoms (96 slots, 48 blocks)
// 77 us per CG iteration, against 16 us for this kernel (28 MB read by 36,864
// threads; both under ncu, cold) and 5 us for the consumer.  One FP64
// evaluation there went from 7.03 to 6.65 ms.
__global__ void k_slot_sum(size_t count, int nslot, double* __restrict__ partial) {
    const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    double s = 0.0;
#pragma unroll 8
    for (int j = 0; j < nslot; j++) s += partial[(size_t)j * count + k];
    partial[k] = s;
}

void slot_sum(const Dev& d, int ncomp, cudaStream_t st) {
    if (d.pp.n_bands < 2) return;
    const size_t count = (size_t)ncomp * d.n_pad;
    k_slot_sum<<<(unsigned)((count + 127) / 128), 128, 0, st>>>(count, d.pp.n_bands, d.partial);
}

}  // namespace

// kind 0: permanent field (operand: the lab dipoles); kind 1: mutual-field
// matvec (operand: vec); kind 2: the start of a warm-started solve, the
// permanent field plus T mu0 in one walk (operand vec = m + mu0, see
// add_partner).
template <>
void launch_field<float>(const Dev& d, int kind, cudaStream_t st, CgStop stop) {
    const int L = d.field_L, B = std::max(L, kFieldNS), nb = (d.pp.n_tiles + B - 1) / B;
    const dim3 grid((unsigned)((long)nb * (nb + 1) / 2 * (B / std::min(L, kFieldNS))), d.field_parts);
    const float4 *pq = (const float4*)d.posq_s, *op = (const float4*)(kind == 0 ? d.dipt_s : d.vec_s);
    const unsigned blocks = (unsigned)((d.n_pad + 127) / 128);
    if (kind == 1) {
        launch_cg_matvec(d, stop, st);
        k_field_done<1><<<blocks, 128, 0, st>>>(d.pp, 0, pq, op, nullptr, d.pos_s, d.exs_off, d.exs_j, d.exs_m,
                                                d.exs_s, d.n_pad, d.fixacc, 1.0 / d.fix_scale, d.partial);
    } else {
        k_field_items<0, kFieldNS><<<grid, 32, 0, st>>>(d.pp, L, pq, op, d.tctr_s, d.text_s, d.pos_s, d.exs_off,
                                                        d.exs_j, d.exs_m, d.exs_tiles, d.n_pad, fix_of(d), stop);
        k_field_done<0><<<blocks, 128, 0, st>>>(d.pp, kind == 2 ? 1 : 0, pq, op, (const float4*)d.dipt_s, d.pos_s,
                                                d.exs_off, d.exs_j, d.exs_m, d.exs_s, d.n_pad, d.fixacc,
                                                1.0 / d.fix_scale, d.partial);
    }
}

template <>
void launch_field<double>(const Dev& d, int kind, cudaStream_t st, CgStop stop) {
    const int BT = d.field_L, nb = (d.pp.n_tiles + BT - 1) / BT;
    const dim3 grid((unsigned)(nb * (nb + 1) / 2), d.field_parts);
    const size_t smem = field_smem(BT);
    const double4 *pq = (const double4*)d.posq_s, *op = (const double4*)(kind == 0 ? d.dipt_s : d.vec_s);
    if (kind == 1) {
        cudaFuncSetAttribute(k_field_bands<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        k_field_bands<1><<<grid, 16 * BT, smem, st>>>(d.pp, BT, pq, op, d.tctr_s, d.text_s, d.exs_off, d.exs_j,
                                                      d.exs_s, d.exs_tiles, d.n_pad, d.partial, stop);
        k_field_slots<1><<<d.n_pad / 32, 96, 0, st>>>(d.pp, 0, pq, op, nullptr, d.pos_s, d.exs_off, d.exs_j, d.exs_m,
                                                      d.exs_s, d.n_pad, nb * d.field_parts, d.partial, stop);
    } else {
        cudaFuncSetAttribute(k_field_bands<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        k_field_bands<0><<<grid, 16 * BT, smem, st>>>(d.pp, BT, pq, op, d.tctr_s, d.text_s, d.exs_off, d.exs_j,
                                                      d.exs_m, d.exs_tiles, d.n_pad, d.partial, stop);
        k_field_slots<0><<<d.n_pad / 32, 96, 0, st>>>(d.pp, kind == 2 ? 1 : 0, pq, op, (const double4*)d.dipt_s,
                                                      d.pos_s, d.exs_off, d.exs_j, d.exs_m, d.exs_s, d.n_pad,
                                                      nb * d.field_parts, d.partial, stop);
    }
}

// The cluster form of the CG kernels holds up to four atoms a thread.  With one
// atom a thread it also collects the mixed matvec's sums; beyond, the partner
// pairs of several atoms in a row would take longer than k_field_done (26 us
// an iteration, cold, against 18 + 6 at 12,288 atoms).
bool cg_cluster(const Dev& d) { return d.n <= 4 * kCgCap; }
bool cg_collects(const Dev& d) { return d.n <= kCgCap; }

namespace {

// Threads of a CTA: one atom each up to kCgThreads, the atoms spread over all
// eight CTAs, so that the partner pairs use all eight SMs and the sums fewer
// warps (an evaluation with CTAs of 512 threads and with these: 286 and 270 us
// at 648 atoms, mixed, 467 and 453 at 1,029, FP64).  Beyond, a thread's further
// atoms lie kCgCap apart.
int cg_threads(const Dev& d) { return std::min(kCgThreads, (d.n_pad + 32 * kCgCtas - 1) / (32 * kCgCtas) * 32); }

CgArrays cg_arrays(const Dev& d, int slot, double* host_eps) {
    CgArrays A{};
    A.order = d.order;
    A.partial = d.partial;
    A.salpha = d.salpha;
    A.thole = d.thole;
    A.E = d.E;
    A.y = d.y;
    A.r = d.r;
    A.p = d.p;
    A.scal_rr = d.scal_rr;
    A.scal_eps = d.scal_eps;
    A.host_eps = host_eps;
    A.n = d.n;
    A.n_pad = d.n_pad;
    A.slot = slot;
    return A;
}

}  // namespace

template <class R>
void launch_cg_start(const Dev& d, int slot, bool use_partial, double* host_eps, cudaStream_t st) {
    const CgArrays A = cg_arrays(d, slot, host_eps);
    k_cg_start<R, 4><<<kCgCtas, cg_threads(d), 0, st>>>(A, (typename Vec4T<R>::type*)d.vec_s, use_partial ? 1 : 0);
}
template void launch_cg_start<float>(const Dev&, int, bool, double*, cudaStream_t);
template void launch_cg_start<double>(const Dev&, int, bool, double*, cudaStream_t);

// Mixed all-pairs matvec without the collection of its sums, which
// launch_cg_step does.
void launch_cg_matvec(const Dev& d, CgStop stop, cudaStream_t st) {
    const int L = d.field_L, B = std::max(L, kFieldNS), nb = (d.pp.n_tiles + B - 1) / B;
    const dim3 grid((unsigned)((long)nb * (nb + 1) / 2 * (B / std::min(L, kFieldNS))), d.field_parts);
    k_field_items<1, kFieldNS><<<grid, 32, 0, st>>>(d.pp, L, (const float4*)d.posq_s, (const float4*)d.vec_s, d.tctr_s,
                                                    d.text_s, d.pos_s, d.exs_off, d.exs_j, d.exs_s, d.exs_tiles,
                                                    d.n_pad, fix_of(d), stop);
}

template <class R>
void launch_cg_step(const Dev& d, int slot, bool collect, CgStop stop, double* host_eps, cudaStream_t st) {
    CgArrays A = cg_arrays(d, slot, host_eps);
    A.stop = stop;
    typedef typename Vec4T<R>::type V4;
    const V4* pq = (const V4*)d.posq_s;
    V4* vec = (V4*)d.vec_s;
    const int threads = cg_threads(d);
#define TDP_CG_STEP(DONE, M)                                                                                       \
    k_cg_step<R, DONE, M><<<kCgCtas, threads, 0, st>>>(d.pp, A, pq, vec, d.pos_s, d.exs_off, d.exs_j, d.exs_m, \
                                                          d.exs_s)
    if constexpr (sizeof(R) == 4)
        if (collect) {
            A.acc = d.fixacc;
            A.inv_scale = 1.0 / d.fix_scale;
            TDP_CG_STEP(true, 1);
            return;
        }
    if (d.n <= kCgCap) TDP_CG_STEP(false, 1);
    else if (d.n <= 2 * kCgCap) TDP_CG_STEP(false, 2);
    else TDP_CG_STEP(false, 4);
#undef TDP_CG_STEP
}
template void launch_cg_step<float>(const Dev&, int, bool, CgStop, double*, cudaStream_t);
template void launch_cg_step<double>(const Dev&, int, bool, CgStop, double*, cudaStream_t);

template <>
void launch_energy<float>(const Dev& d, cudaStream_t st) {
    const int L = d.energy_L, nb = (d.pp.n_tiles + L - 1) / L;
    const dim3 grid((unsigned)((long)nb * (nb + 1) / 2 * L), d.energy_parts);
    const float4 *pq = (const float4*)d.posq_s, *dp = (const float4*)d.dipt_s, *u = (const float4*)d.vec_s;
    FixAcc fix = fix_of(d);
    fix.scale = d.fix_scale_energy;
    const IndexRecords rec{(const float4*)d.posq, d.tctr, pq, dp, u};
    const EItemArrays A{pq, dp, u, d.order, d.tctr_s, d.text_s, d.pos_s, d.exs_off, d.exs_j, d.exs_m, d.exs_s,
                        d.exs_tiles, rec, AxisList{d.axis_pairs, d.axis_count, (unsigned long long)d.axis_cap}, fix, L,
                        d.n_pad};
    if (d.pp.lab_energy && !d.pp.periodic) k_energy_items<false, true><<<grid, 32, 0, st>>>(d.pp, A, d.energy_partial);
    else if (d.pp.lab_energy) k_energy_items<false, false><<<grid, 32, 0, st>>>(d.pp, A, d.energy_partial);
    else k_energy_items<true, false><<<grid, 32, 0, st>>>(d.pp, A, d.energy_partial);
    k_axis_pairs<<<std::min(8 * 148, std::max(148, d.pp.n_tiles)), 32, 0, st>>>(d.pp, A, (int)grid.x);
    k_energy_items_done<<<d.n_pad / 128, 128, 0, st>>>(d.pp, pq, dp, u, d.order, d.pos_s, d.exs_off, d.exs_j, d.exs_m,
                                                       d.exs_s, rec, d.axis_count, d.n_pad, d.fixacc,
                                                       1.0 / fix.scale, d.n_eblk,
                                                       d.energy_partial, d.fpair, d.torque,
                                                       d.energy_partial + d.n_eblk);
    launch_energy_total(d, d.n_pad / 128, d.energy_partial + d.n_eblk, st);
}

template <>
void launch_energy<double>(const Dev& d, cudaStream_t st) {
    const size_t smem = energy_smem(d.pp.band_tiles);
    cudaFuncSetAttribute(k_energy_sym, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_energy_sym<<<band_pairs(d), 32 * std::min(kSymWarps, d.pp.band_tiles), smem, st>>>(
        d.pp, (const double4*)d.posq, (const double4*)d.dipt, (const double4*)d.ind, d.yz, d.tctr, d.text, d.pos,
        d.exc_off, d.exc_j, d.exc_m, d.exc_s, d.exc_tiles, d.n_pad, d.partial, d.energy_partial);
    slot_sum(d, 6, st);
    launch_energy_done(d, st);
}

}  // namespace tdp
