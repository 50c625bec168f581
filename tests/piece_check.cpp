// Host check of the certified pieces (csrc/cpd_piece.h) against fast_ray, ray by ray.
//
// For every wavelength of the given points the core range is cut into pieces as the device
// cuts it; every ray that a piece decides must get from fast_ray the same outcome, the same
// bin and, on a hit, the wavelength's transmittance, and no flag.
//
// usage: piece_check design.bin W R lam_u.bin ray_u.bin
// prints: rays <core rays> decided <by a piece> wrong <disagreements> edge <rays a quadratic left to
//         fast_ray> whole <rays of pieces left to fast_ray> mixed <rays decided by a quadratic> pieces <n>
//         by_edges <rays of pieces binned by their edges>
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "cpd_df.h"
#include "cpd_host.h"
#include "cpd_piece.h"

using namespace cpd;

static std::vector<double> read(const char *path, int n)
{
    std::vector<double> v(n);
    FILE *f = std::fopen(path, "rb");
    if (!f || std::fread(v.data(), 8, n, f) != (size_t)n) std::exit(3);
    std::fclose(f);
    return v;
}

int main(int argc, char **argv)
{
    if (argc < 6) return 2;
    cpd_design d;
    FILE *f = std::fopen(argv[1], "rb");
    if (!f || std::fread(&d, sizeof d, 1, f) != 1) return 3;
    std::fclose(f);
    const int W = std::atoi(argv[2]), R = std::atoi(argv[3]);
    const std::vector<double> lu = read(argv[4], W), ru = read(argv[5], R);
    DevDesign D;
    design_to_dev(d, D);
    std::vector<double> z64;
    std::vector<float> z32;
    ray_table(ru.data(), R, z64, z32);
    const Guards g = default_guards();
    const FastLimits Lm = fast_limits(D.fc, g);
    const PieceConst K = piece_const(D.fc);
    long rays = 0, decided = 0, wrong = 0, edge = 0, whole = 0, mixed = 0, pieces = 0, by_edges = 0;
    for (int k = 0; k < W; k++) {
        LamParams P;
        LamDF E;
        lambda_setup_df(D, lu[k], z32.data(), (uint32_t)z64.size(), P, kYGuardRel, &E);
        if (P.all_exact || P.core_hi <= P.core_lo) continue;
        const uint32_t lo = P.core_lo, hi = P.core_hi, n = hi - lo, L = (n + 14u) / 15u;
        const uint32_t T = piece_tfix(P);
        rays += n;
        for (uint32_t j0 = lo; j0 < hi; j0 += L) {
            const uint32_t j1 = j0 + L < hi ? j0 + L : hi, jb = j0 + L < hi ? j0 + L : hi - 1u;
            const PieceEnd a = piece_end(D.fc, Lm, K, P, g, z32[2 * j0], z32[2 * j0 + 1]);
            const PieceEnd b = piece_end(D.fc, Lm, K, P, g, z32[2 * jb], z32[2 * jb + 1]);
            Piece q = piece_fit(D.fc, K, P, a, b);
            if (!D.fc.pieces) q.cls = PIECE_RAYS;
            pieces++;
            // the same piece as one quadratic for piece_ray (adaptive sampling)
            {
                const Piece u = piece_uniform(K, q);
                for (uint32_t j = j0; j < j1; j++) {
                    const float dz = (P.zref_hi - z32[2 * j]) + (P.zref_lo - z32[2 * j + 1]);
                    uint32_t bin = 0;
                    const int r = piece_ray(K, D.B, u.dz0, u.v0, u.v1, u.v2, u.e, dz, bin);
                    const int want = q.cls == PIECE_BIN ? RAY_HIT : q.cls == PIECE_LOST ? RAY_LOST : RAY_FLAG;
                    if (q.cls != PIECE_MIXED && (r != want || (r == RAY_HIT && bin != q.bin))) wrong++;
                }
            }
            // the outcome of every ray of the piece: its bin, -1 lost, -2 left to fast_ray
            std::vector<int> out(j1 - j0, q.cls == PIECE_BIN ? (int)q.bin : q.cls == PIECE_LOST ? -1 : -2);
            if (q.cls == PIECE_RAYS) whole += j1 - j0;
            if (q.cls == PIECE_MIXED) {
                const auto dz_of = [&](uint32_t j) { return (P.zref_hi - z32[2 * j]) + (P.zref_lo - z32[2 * j + 1]); };
                const PieceEdges pe = piece_edges(K, q, b.dz - a.dz, L);
                for (uint32_t j = j0; j < j1 && !pe.count; j++) {
                    uint32_t bin = 0;
                    const int r = piece_ray(K, D.B, q.dz0, q.v0, q.v1, q.v2, q.e, dz_of(j), bin);
                    out[j - j0] = r == RAY_HIT ? (int)bin : r == RAY_LOST ? -1 : -2;
                }
                if (pe.count) {
                    by_edges += j1 - j0;
                    std::fill(out.begin(), out.end(), -1);
                }
                for (uint32_t t = 0; t < pe.count; t++) {
                    const bool ext = pe.ext && t + 1u == pe.count;
                    const int bq = pe.qa + (int)t;
                    const float sg = q.v1 > 0.f ? -1.f : 1.f;
                    EdgeRays r[2];
                    for (int up = 0; up < 2; up++) {
                        const Edge ed = piece_edge(K, bq, ext, up);
                        const float a0 = sg * (q.v0 - ed.v), a1 = sg * q.v1, a2 = sg * q.v2;
                        r[up] = edge_rays(j0, j1, q.e, [&](uint32_t j) {
                            const float dd = dz_of(j) - q.dz0;
                            return a0 + dd * (a1 + dd * a2);
                        });
                        for (uint32_t j = r[up].jb; j < r[up].je && ed.emit; j++) {
                            if (out[j - j0] == -2) wrong++;  // listed twice
                            out[j - j0] = -2;
                        }
                    }
                    const uint32_t first = sg > 0.f ? r[0].je : r[1].je, last = sg > 0.f ? r[1].jb : r[0].jb;
                    const uint32_t bin = bq > 0 ? (uint32_t)bq : 0u;
                    for (uint32_t j = first; j < last && !ext && bin < D.B; j++) {
                        if (out[j - j0] != -1) wrong++;
                        out[j - j0] = (int)bin;
                    }
                }
                for (const int o : out) (o == -2 ? edge : mixed)++;
            }
            for (uint32_t j = j0; j < j1; j++) {
                const int o = out[j - j0];
                if (o == -2) continue;
                decided++;
                uint32_t bf = 0;
                float tf = 0.f;
                const int rf = fast_ray(D.fc, Lm, P, g, z32[2 * j], z32[2 * j + 1], bf, tf);
                if (rf != (o >= 0 ? RAY_HIT : RAY_LOST) || (o >= 0 && ((int)bf != o || t_fixed(tf) != T))) wrong++;
            }
        }
    }
    std::printf("rays %ld decided %ld wrong %ld edge %ld whole %ld mixed %ld pieces %ld by_edges %ld\n",
                rays, decided, wrong, edge, whole, mixed, pieces, by_edges);
    return 0;
}
