// cpd_piece.h -- a wavelength's detector coordinate as certified quadratics of the start height.
//
// Every ray of one wavelength meets the exit face with the same direction d, and its offset
// from the face's centre across d, x = sin(theta) Rc, is affine in the start height. So the
// detector coordinate pos is a closed-form function of one variable, and with
//   theta_r = asin(r x), kappa = r cos(theta)/cos(theta_r)     (refraction into air, r = n)
//   psi the exit direction's angle from the detector's normal, psi' = 1 - kappa
//   T the distance travelled to the detector line
// its derivatives along theta are (eps = +-1 the detector's orientation)
//   pos'  = eps sec(psi) A,          A  = Rc cos(theta_r) - T (kappa - 1)
//   pos'' = eps sec(psi) B,          B  = -Rc sin(theta_r) (2 kappa - 1) - 2 A (kappa - 1) tan(psi) - T kappa'
//   kappa' = kappa (kappa tan(theta_r) - tan(theta)),  T' = Rc sin(theta_r) + A tan(psi)
// (and pos''' by the product rule). Over a piece of consecutive rays every factor is bounded
// by its values at the two ends (theta_r and kappa grow with |x|, psi is monotone), so
// |pos'''| has a bound, and the quadratic through both ends' coordinates with the first end's
// slope is within 4/27 H^3/6 max|pos'''| of pos. With an anti-reflection coated exit face
// (cos(theta) > 0.5 throughout the piece) the transmittance is the same for every ray of the
// wavelength, so a ray's bin is all that is left to know: it comes from the quadratic wherever
// that is further from a bin edge than its error bound plus twice the fast path's own guard.
// The other rays (a few per wavelength) are left to fast_ray. A piece whose ends do not both
// clear, or both fail in the same way, every test of fast_ray by twice its guard is left to
// fast_ray whole. So every ray gets the bin, the transmittance or the flag that fast_ray gives
// it (tests/piece_check.cpp compares them ray by ray).
#pragma once

#include "cpd_model.h"

// A mixed piece's bins come from its edges when it has at least this many rays per bin it
// crosses: finding two edges by bisection costs about as much as binning that many rays.
#ifndef CPD_EDGE_RAYS
#define CPD_EDGE_RAYS 4
#endif

namespace cpd {

// Design constants of the pieces, in bins: v = (pos - c0)/slope - 1/2, so that the bin is v
// rounded to nearest and the remainder lies in [-1/2, 1/2].
struct PieceConst {
    float vmid, vhalf;  // the detector's extent [0, L]: |v - vmid| <= vhalf
    float fs;           // a remainder below fs is on the bin's sensitive part
    float rc;           // exit-face radius
    float eps;          // +-1: -(N x U)
    float sep, sepx;    // smallest distance between two bin edges, and between a bin edge and the extent's ends
};
// v rounded to nearest (|v| < 2^22): the sum's low bits are the integer.
CPD_HD float round_bin(float v) { return ff::sub_rn(ff::add_rn(v, 12582912.f), 12582912.f); }
// Distance of v from the nearest bin edge (q - 1/2 or q + fs).
CPD_HD float edge_distance(const PieceConst &K, float v)
{
    const float r = v - round_bin(v), a = 0.5f - fabs_f(r), b = fabs_f(r - K.fs);
    return a < b ? a : b;
}
CPD_HD PieceConst piece_const(const FastConst &D)
{
    PieceConst c;
    c.vhalf = D.hL * D.inv_slope;
    c.vmid = (D.hL - D.c0) * D.inv_slope - 0.5f;
    c.fs = D.bin_size * D.inv_slope - 0.5f;
    c.rc = 1.f / D.inv_rc;
    c.eps = D.dnfy * D.dufx - D.dnfx * D.dufy;
    const float on = c.fs + 0.5f, gap = 0.5f - c.fs;
    c.sep = on < gap ? on : gap;  // negative when the bins overlap
    c.sepx = edge_distance(c, c.vmid - c.vhalf);
    const float hi = edge_distance(c, c.vmid + c.vhalf);
    if (hi < c.sepx) c.sepx = hi;
    return c;
}

// How a ray at a piece's end fares, by twice fast_ray's guards.
enum : int {
    END_CLEAR = 0,                       // clears every test before the detector coordinate
    END_APERTURE = 1,                    // outside the exit face's bound
    END_TIR_POS = 2, END_TIR_NEG = 3,    // total internal reflection, x > 0 or x < 0
    END_WEAK_POS = 4, END_WEAK_NEG = 5,  // too oblique on the detector, exit direction along U or against it
    END_UNSURE = 6
};
struct PieceEnd {
    float dz;              // zref - z
    float v, gv;           // detector coordinate and fast_ray's guard there, in bins
    float slope;           // dv/d(dz)
    float ci, cr, cid;     // cosines: exit face in and out, detector
    float gn;              // distance to the detector's line along its normal
    float px, py;          // hit point relative to the bound's centre
    int cls;
};

// fast_ray's quantities at one start height.
CPD_HD PieceEnd piece_end(const FastConst &D, const FastLimits &Lm, const PieceConst &K, const LamParams &P,
                          const Guards &g, float zhi, float zlo)
{
    PieceEnd e;
    const float dz = (P.zref_hi - zhi) + (P.zref_lo - zlo);
    e.dz = dz;
    const float dud = P.uz * dz;
    const float ddisc = dud * (P.ud2 + dud) - dz * (P.cb * dz + P.ca);
    const float disc = P.disc + ddisc;
    const float sd = sqrt_fast(disc > 0.f ? disc : 0.f);
    const float ds = P.sigma * div_fast(ddisc, sd + P.sd) - dud;
    const float s = P.s + ds;
    const float dpx = P.dx * ds + P.wzx * dz, dpy = P.dy * ds + P.wzy * dz;
    e.px = 0.5f * P.px2 + dpx;
    e.py = 0.5f * P.py2 + dpy;
    const float mb = P.mb + (dpx * (P.px2 + dpx) + dpy * (P.py2 + dpy));
    const float dci = (ds + dud) * D.inv_rc;
    e.ci = P.ci + dci;
    const float dcr2 = P.r2 * dci * (P.ci2 + dci);
    const float crsq = P.crsq + dcr2;
    e.cr = sqrt_fast(crsq > 1e-12f ? crsq : 1e-12f);
    const float dkk = P.r * dci - div_fast(dcr2, e.cr + P.cr);
    const float dgn = dpx * D.dnfx + dpy * D.dnfy, dgu = dpx * D.dufx + dpy * D.dufy;
    const float kn = (P.kk + dkk) * D.inv_rc;
    const float dcid = dgn * kn - dkk * P.nf;
    e.cid = P.cid + dcid;
    const float ddu = dkk * P.nu - dgu * kn;
    const float icid = div_fast(1.f, e.cid);
    const float dT = (dgn - P.T * dcid) * icid;
    const float T = P.T + dT;
    const float tu = ddu * T, tt = P.du * dT;
    const float pos = P.pos + (tu + (tt + dgu));
    e.gn = T * e.cid;
    e.v = (pos - D.c0) * D.inv_slope - 0.5f;
    e.gv = (g.pos_rel * (fabs_f(tu) + fabs_f(tt) + fabs_f(dgu) + fabs_f(P.pos)) + g.pos) * D.inv_slope;
    const float kt = div_fast(P.r * e.ci, e.cr) - 1.f;
    e.slope = K.eps * (K.rc * e.cr - T * kt) * div_fast(icid, e.ci) * P.xz * D.inv_slope;
    const float c2 = 2.f * g.cosine;
    int cls = END_UNSURE;
    if (disc > 2.f * g.rel * P.disc && sd > 1.001f * Lm.rho101 && s > 2.f * g.dist) {
        if (mb > 2.f * Lm.rho2g) {
            cls = END_APERTURE;
        } else if (mb < -2.f * Lm.rho2g) {
            if (crsq < -c2) {
                cls = P.xref + P.xz * dz > 0.f ? END_TIR_POS : END_TIR_NEG;
            } else if (crsq > c2 && e.ci > 0.5f + c2) {
                if (e.cid < D.min_ci - c2) cls = P.du + ddu > 0.f ? END_WEAK_POS : END_WEAK_NEG;
                else if (e.cid > D.min_ci + c2 && e.cid > 0.01f) cls = END_CLEAR;
            }
        }
    }
    e.cls = cls;
    return e;
}

// What is known of all rays of a piece.
enum : int { PIECE_LOST = 0, PIECE_BIN = 1, PIECE_MIXED = 2, PIECE_RAYS = 3 };
struct Piece {
    float dz0, v0, v1, v2;  // v = v0 + d (v1 + d v2), d = dz - dz0
    float e;                // bins: within e of an edge, fast_ray decides
    uint32_t bin;           // PIECE_BIN
    int cls;
};

// The rays between the ends a and b.
CPD_HD Piece piece_fit(const FastConst &D, const PieceConst &K, const LamParams &P, const PieceEnd &a,
                       const PieceEnd &b)
{
    Piece q;
    q.cls = PIECE_RAYS;
    q.dz0 = a.dz;
    q.v0 = a.v;
    q.v1 = q.v2 = q.e = 0.f;
    q.bin = 0u;
    const float H = b.dz - a.dz, hx = fabs_f(P.xz * H);
    const float cim = a.ci < b.ci ? a.ci : b.ci;
    const float ici = div_fast(1.f, cim), dth = hx * ici;  // the piece's extent in theta is at most dth
    // sigma < 0 or r < 1: not the geometry the bounds are made for
    if (a.cls != b.cls || a.cls == END_UNSURE || !(P.sigma > 0.f) || !(P.r >= 1.f)) return q;
    if (a.cls == END_APERTURE) {
        // both outside, on the same side of the bound's arc: its two sides are seen from its
        // centre under more than a right angle
        if (cim > 0.1f && dth < 0.5f && a.px * b.px + a.py * b.py > 0.f) q.cls = PIECE_LOST;
        return q;
    }
    if (a.cls == END_TIR_POS || a.cls == END_TIR_NEG) {
        q.cls = PIECE_LOST;  // |x| > 1/r throughout
        return q;
    }
    const float crm = a.cr < b.cr ? a.cr : b.cr;
    const float icr = div_fast(1.f, crm), kap = P.r * cim * icr, kt = kap - 1.f;
    if (!(kt * dth < 0.5f)) return q;
    if (a.cls != END_CLEAR) {
        q.cls = PIECE_LOST;  // psi is monotone: oblique to the same side throughout
        return q;
    }
    // bounds over the piece
    const float cdm = a.cid < b.cid ? a.cid : b.cid;
    const float sec = div_fast(1.f, cdm);
    const float tau2 = ici * ici - 1.f, ttr2 = icr * icr - 1.f, tps2 = sec * sec - 1.f;
    const float tau = sqrt_fast(tau2 > 0.f ? tau2 : 0.f), ttr = sqrt_fast(ttr2 > 0.f ? ttr2 : 0.f);
    const float tps = sqrt_fast(tps2 > 0.f ? tps2 : 0.f);
    const float ga = fabs_f(a.gn), gb = fabs_f(b.gn);
    const float T = ((ga > gb ? ga : gb) + K.rc * dth) * sec;
    const float S = K.rc * ttr * crm, A = K.rc + T * kt;
    const float kap2 = kap * kap, k1 = kap2 * ttr, k2 = 2.f * k1 * kap * ttr + kap * kap2 * (1.f + ttr2);
    const float w = S * (2.f * kap - 1.f) + T * k1, ak = A * kt * tps;
    const float A1 = w + ak, B2 = w + 2.f * ak, T1 = S + A * tps;
    const float B3 = K.rc * kap * (2.f * kap - 1.f) + 2.f * S * k1 + 2.f * tps * (A1 * kt + A * k1) +
                     2.f * A * kt * kt * sec * sec + T1 * k1 + T * k2 + B2 * kt * tps;
    const float M3 = sec * (B3 + 3.f * tau * B2 + (1.f + 3.f * tau2) * A) * (ici * ici * ici);
    const float E = 0.0252f * M3 * (hx * hx * hx) * D.inv_slope;
    // the quadratic, and its rounding
    const float dv = b.v - a.v, sH = a.slope * H;
    q.v1 = a.slope;
    const float c2 = dv - sH;  // v2 H^2
    q.v2 = H != 0.f ? div_fast(c2, H * H) : 0.f;
    const float gm = a.gv > b.gv ? a.gv : b.gv;
    q.e = 2.f * gm + E + 9.5367431640625e-07f * (fabs_f(a.v) + 2.f * fabs_f(sH) + 2.f * fabs_f(c2));
    if (!(q.e < 0.2f)) {
        // too coarse to decide bins; far from the detector it still decides the piece
        if (!(q.e < 1e6f)) return q;
    }
    const float dev = 0.25f * fabs_f(c2) + q.e;  // the quadratic is within c2/4 of its chord
    const float lo = (a.v < b.v ? a.v : b.v) - dev, hi = (a.v < b.v ? b.v : a.v) + dev;
    if (lo - K.vmid > K.vhalf || K.vmid - hi > K.vhalf) {
        q.cls = PIECE_LOST;
        return q;
    }
    if (!(q.e < 0.2f) || !(fabs_f(a.v) < 1e6f) || !(fabs_f(b.v) < 1e6f)) return q;
    q.cls = PIECE_MIXED;
    const float bl = round_bin(lo), bh = round_bin(hi);
    if (bl == bh && K.vmid - lo < K.vhalf && hi - K.vmid < K.vhalf) {
        const float rl = lo - bl, rh = hi - bh;
        if (rl >= K.fs) {
            q.cls = PIECE_LOST;
        } else if (rh < K.fs) {
            const uint32_t bin = bl > 0.f ? (uint32_t)bl : 0u;
            q.cls = bin < D.B ? PIECE_BIN : PIECE_LOST;
            q.bin = bin;
        }
    }
    return q;
}

// One ray of a mixed piece: RAY_HIT with its bin, RAY_LOST, or RAY_FLAG: fast_ray decides.
CPD_HD int piece_ray(const PieceConst &K, uint32_t B, float dz0, float v0, float v1, float v2, float e, float dz,
                     uint32_t &bin)
{
    const float d = dz - dz0;
    const float v = v0 + d * (v1 + d * v2);
    const float bf = ff::add_rn(v, 12582912.f);
    const float r = v - ff::sub_rn(bf, 12582912.f);
    const float off = fabs_f(v - K.vmid) - K.vhalf;
    if (off > e) return RAY_LOST;
    if ((off > -e) | (fabs_f(r) > 0.5f - e) | (fabs_f(r - K.fs) < e)) return RAY_FLAG;
#if defined(__CUDA_ARCH__)
    const int b = (int)(__float_as_uint(bf) - 0x4B400000u);
#else
    const int b = (int)(bf - 12582912.f);
#endif
    bin = b > 0 ? (uint32_t)b : 0u;
    return (r < K.fs && bin < B) ? RAY_HIT : RAY_LOST;
}

// The edges of a mixed piece of len rays, as tasks: task k is the two edges q - 1/2 and q + fs
// of bin q = qa + k, and with `ext` one more task the two ends of the detector's extent.
// count 0: the rays are to be binned one by one (the coordinate turns within the piece, or
// edges lie too close together for the error bound, or too many for the rays they save).
struct PieceEdges {
    int qa;
    uint32_t count;
    bool ext;
};
CPD_HD PieceEdges piece_edges(const PieceConst &K, const Piece &q, float H, uint32_t len)
{
    PieceEdges t;
    t.qa = 0;
    t.count = 0u;
    t.ext = false;
    const float s1 = q.v1 + 2.f * q.v2 * H;
    if (!((q.v1 > 0.f && s1 > 0.f) || (q.v1 < 0.f && s1 < 0.f)) || !(4.f * q.e < K.sep)) return t;
    const float vb = q.v0 + H * (q.v1 + H * q.v2);
    float lo = (q.v0 < vb ? q.v0 : vb) - 2.f * q.e, hi = (q.v0 < vb ? vb : q.v0) + 2.f * q.e;
    const float xlo = K.vmid - K.vhalf, xhi = K.vmid + K.vhalf;
    t.ext = lo < xlo || hi > xhi;
    if (t.ext && !(4.f * q.e < K.sepx)) return t;
    if (lo < xlo) lo = xlo;
    if (hi > xhi) hi = xhi;
    const float qa = round_bin(lo), qb = round_bin(hi);
    const float n = qb - qa + 1.f + (t.ext ? 1.f : 0.f);
    if (!(n >= 1.f) || n * (float)CPD_EDGE_RAYS > (float)len) return t;
    t.qa = (int)qa;
    t.count = (uint32_t)n;
    return t;
}

// One edge of a task: lower (q - 1/2, or the extent's lower end) or upper (q + fs, its upper
// end). A bin's edge beyond the extent's end is that end; the extent's own task then emits its
// rays for fast_ray.
struct Edge {
    float v;
    bool emit;
};
CPD_HD Edge piece_edge(const PieceConst &K, int q, bool ext, bool up)
{
    const float x = up ? K.vmid + K.vhalf : K.vmid - K.vhalf;
    if (ext) return Edge{x, true};
    const float v = up ? (float)q + K.fs : (float)q - 0.5f;
    return (up ? v <= x : v >= x) ? Edge{v, true} : Edge{x, false};
}

// The rays [jb, je) of [p0, p1) within e of an edge, by bisection: at(j) is ray j's v less the
// edge's, with the sign that makes it rise with j. Rays before jb and from je on lie on their side
// of the edge. The bracket keeps both ends' values, so that the window costs nothing more unless a
// ray is in it.
struct EdgeRays {
    uint32_t jb, je;
};
template <class At>
CPD_HD EdgeRays edge_rays(uint32_t p0, uint32_t p1, float e, const At &at)
{
    uint32_t lo = p0 - 1u, hi = p1;  // at(lo) < 0 <= at(hi); the ends stand outside the piece
    float alo = -1e30f, ahi = 1e30f;
    while (hi - lo > 1u) {
        const uint32_t m = lo + ((hi - lo) >> 1);
        const float a = at(m);
        const bool before = a < 0.f;
        lo = before ? m : lo;
        alo = before ? a : alo;
        hi = before ? hi : m;
        ahi = before ? ahi : a;
    }
    EdgeRays r;
    r.jb = r.je = hi;
    if (-alo < e) {
        r.jb = lo;
        while (r.jb > p0 && fabs_f(at(r.jb - 1u)) < e) r.jb--;
    }
    if (ahi < e) {
        r.je = hi + 1u;
        while (r.je < p1 && fabs_f(at(r.je)) < e) r.je++;
    }
    return r;
}

// log2 of the rays per piece that cut n rays into at most 31 pieces (32 ends).
CPD_HD uint32_t piece_shift(uint32_t n)
{
    uint32_t k = 0;
    while ((31u << k) < n) k++;
    return k;
}

// A piece as a quadratic and an error that make piece_ray give every ray the piece's outcome: a
// piece in one bin or lost whole is a constant in the bin's sensitive part or off the detector, a
// piece without a bound has an error beyond every bin.
CPD_HD Piece piece_uniform(const PieceConst &K, Piece q)
{
    if (q.cls == PIECE_MIXED) return q;
    q.v1 = q.v2 = q.e = 0.f;
    q.v0 = q.cls == PIECE_BIN ? (float)q.bin + 0.5f * ((K.fs < 0.5f ? K.fs : 0.5f) - 0.5f)
                              : K.vmid + 2.f * K.vhalf + 1.f;
    if (q.cls == PIECE_RAYS) q.e = 1e30f;
    return q;
}

// 2^31 t of every hit of a certified piece: fast_ray's coated transmittance.
CPD_HD uint32_t piece_tfix(const LamParams &P) { return t_fixed(mulr(addr(P.ts, P.tp), 0.495f)); }

}  // namespace cpd
