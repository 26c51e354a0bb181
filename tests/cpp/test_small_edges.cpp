// Host check of the setup kernel's small-triangle path (fr_exact.cuh: small_edges,
// box_row, bary_off_edge, bary_on_edge) against bary<0, false> on every pixel of the
// clamped box: same coverage, same weights; and that box_may_be_covered never drops a
// tile with a covered pixel, for triangles of every class. Exit status 0 = no difference.
// Usage: test_small_edges <num_triangles> <seed>
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "fr_exact.cuh"

int main(int argc, char** argv)
{
    const long n = argc > 1 ? std::atol(argv[1]) : 100000;
    std::mt19937_64 rng(argc > 2 ? std::atoi(argv[2]) : 1);
    long pixels = 0, covered = 0, edge = 0, bad = 0, rows = 0;
    for (long it = 0; it < n; ++it)
    {
        frx::RTri t;
        const int span = (const int[]){1, 3, 8, 20, 60, 400, 16000}[rng() % 7];
        const int W = 1 + (int)(rng() % 8192), H = 1 + (int)(rng() % 8192);
        const int cx = (int)(rng() % (W + 40)) - 20, cy = (int)(rng() % (H + 40)) - 20;
        for (int k = 0; k < 3; ++k)
        {
            t.x[k] = cx + (int)(rng() % (2 * span + 1)) - span;
            t.y[k] = cy + (int)(rng() % (2 * span + 1)) - span;
            t.d[k] = 0.f;
        }
        if (rng() % 8 == 0) t.y[1] = t.y[0];
        if (rng() % 8 == 0) t.x[2] = t.x[1];
        if (rng() % 4 == 0) std::swap(t.x[1], t.x[2]), std::swap(t.y[1], t.y[2]);
        frx::classify(t);
        if (t.cls != frx::kTriFast || !t.small) continue;
        auto cl = [](int v, int hi) { return std::min(hi, std::max(v, 0)); };
        const int x0 = cl(std::min({t.x[0], t.x[1], t.x[2]}), W - 1), x1 = cl(std::max({t.x[0], t.x[1], t.x[2]}), W - 1);
        const int y0 = cl(std::min({t.y[0], t.y[1], t.y[2]}), H - 1), y1 = cl(std::max({t.y[0], t.y[1], t.y[2]}), H - 1);
        const long area = (long)(x1 - x0 + 1) * (y1 - y0 + 1);
        if (area > 65536) continue;
        const int w = x1 - x0 + 1;
        const frx::SmallEdges s = frx::small_edges(t, x0, y0);
        const float rw = 1.f / (float)w, rB = t.rbz < 0.f ? -t.rbz : t.rbz;
        const long step = area > 4096 ? 37 : 1;
        for (long l = 0; l < area; l += step)
        {
            const int ly = frx::box_row((int)l, rw), lx = (int)l - ly * w;
            if (ly != (int)(l / w)) ++bad;
            const int e1 = frx::affine_wrapped(s.a1, s.bx1, s.by1, lx, ly);
            const int e2 = frx::affine_wrapped(s.a2, s.bx2, s.by2, lx, ly);
            const int c = s.B - e1 - e2;
            float g0 = 0, g1 = 0, g2 = 0, r0 = 0, r1 = 0, r2 = 0;
            bool got = (e1 | e2 | c) >= 0;
            if (got && c == 0) ++edge;
            if (got)
                got = c ? frx::bary_off_edge(e1, e2, s.B, rB, g0, g1, g2)
                        : frx::bary_on_edge(e1, e2, s.B, rB, t.m53, t.s53, g0, g1, g2);
            const bool want = frx::bary<0, false>(t, x0 + lx, y0 + ly, r0, r1, r2);
            ++pixels;
            covered += want;
            if (want)
            {
                // a resolve's form, and the edges of the absolute pixel
                float h0, h1, h2;
                frx::bary_covered(t, x0 + lx, y0 + ly, h0, h1, h2);
                const frx::SmallEdges z = frx::small_edges(t, 0, 0);
                if (h0 != r0 || h1 != r1 || h2 != r2 ||
                    frx::affine_wrapped(z.a1, z.bx1, z.by1, x0 + lx, y0 + ly) != e1 ||
                    frx::affine_wrapped(z.a2, z.bx2, z.by2, x0 + lx, y0 + ly) != e2)
                    ++bad;
            }
            // a zero weight's sign is not part of the form (kZeroSigns = false)
            auto same = [](float a, float b) { return std::memcmp(&a, &b, 4) == 0 || (a == 0.f && b == 0.f); };
            if (got != want || (want && !(same(g0, r0) && same(g1, r1) && same(g2, r2))))
            {
                if (bad++ < 10)
                    std::printf("MISMATCH (%d,%d)(%d,%d)(%d,%d) px (%d,%d): %d %a %a %a vs %d %a %a %a\n", t.x[0], t.y[0],
                                t.x[1], t.y[1], t.x[2], t.y[2], x0 + lx, y0 + ly, got, g0, g1, g2, want, r0, r1, r2);
            }
        }
    }
    // 16 x 16 tiles against triangles of every class, many of them with far vertices
    long tiles = 0, kept = 0;
    for (long it = 0; it < n / 2; ++it)
    {
        frx::RTri t;
        const long span = (const long[]){12, 60, 400, 5000, 100000, 9000000, 2000000000}[rng() % 7];
        const int tx = (int)(rng() % 128) * 16, ty = (int)(rng() % 128) * 16;
        for (int k = 0; k < 3; ++k)
        {
            const long s2 = rng() % 3 ? span : 40;
            t.x[k] = (int)std::max(-2147483647l, std::min(2147483647l, tx + (long)(rng() % (2 * s2 + 1)) - s2));
            t.y[k] = (int)std::max(-2147483647l, std::min(2147483647l, ty + (long)(rng() % (2 * s2 + 1)) - s2));
            t.d[k] = 0.f;
        }
        if (rng() % 8 == 0) t.y[1] = t.y[0];
        frx::classify(t);
        if (t.cls == frx::kTriEmpty) continue;
        bool any = false;
        for (int q = 0; q < 256; ++q)
        {
            float b0, b1, b2;
            any = any || frx::bary<0, false>(t, tx + q % 16, ty + q / 16, b0, b1, b2);
        }
        const bool keep = frx::box_may_be_covered(t, tx, tx + 15, ty, ty + 15);
        ++tiles, kept += keep;
        if (any && !keep && bad++ < 10) std::printf("TILE DROPPED class %d\n", t.cls);
    }
    std::printf("tiles %ld kept %ld\n", tiles, kept);
    // every row of every box width a small triangle can have
    for (int w = 1; w <= 8192; w = w < 300 ? w + 1 : w + 61)
        for (int l = 0; l < 65536; l += w < 8 ? 1 : 7, ++rows)
            if (frx::box_row(l, 1.f / (float)w) != l / w) ++bad;
    std::printf("pixels %ld covered %ld on edge %ld rows %ld mismatches %ld\n", pixels, covered, edge, rows, bad);
    return bad == 0 ? 0 : 1;
}
