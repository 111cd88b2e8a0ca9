// Host build of the fixed-point weights (csrc/fx_weight.cuh, csrc/fx_geo.cuh) for the CPU tests.
#include "../../libgwmodel_gb300/csrc/fx_geo.cuh"

using namespace gwgpu::fx;

extern "C" {

// Weight (times 2^62) of a pair at integer coordinate differences (dx, dy) 2^-scale
// for threshold r by the fast (where it applies) or the general arithmetic; ~0 when r is not a positive normal number.
uint64_t fx_weight(int gauss, int general, double r, int scale, int64_t dx, int64_t dy)
{
    static uint64_t table[256];
    if (!table[0])
        for (int i = 0; i < 256; i++) table[i] = exp2_entry(i);
    Row row;
    if (!(gauss ? row_setup<true>(r, scale, row) : row_setup<false>(r, scale, row))) return ~0ull;
    if (!row.limh || general)
        return gauss ? gaussian(dist2<true, false>(dx, dy, row), row, table) : bisquare(dist2<false, false>(dx, dy, row), row);
    return gauss ? gaussian(dist2<true, true>(dx, dy, row), row, table) : bisquare(dist2<false, true>(dx, dy, row), row);
}

// The same for two unit vectors times 2^61 and a threshold in km.
uint64_t fx_geo_weight(int gauss, int general, double r, const int64_t* a, const int64_t* b)
{
    static uint64_t table[256];
    static GeoCoef geo[kGeoIntervals];
    if (!table[0]) {
        geo_table(geo);
        for (int i = 0; i < 256; i++) table[i] = exp2_entry(i);
    }
    Row row;
    if (!(gauss ? geo_row_setup<true>(r, row) : geo_row_setup<false>(r, row))) return ~0ull;
    const Vec3 p{a[0], a[1], a[2], 0}, q{b[0], b[1], b[2], 0};
    if (!row.limh) general = 1;
    const Chord c = gauss ? (general ? geo_chord<true, false>(p, q, row) : geo_chord<true, true>(p, q, row))
                          : (general ? geo_chord<false, false>(p, q, row) : geo_chord<false, true>(p, q, row));
    if (!geo_near(c, row)) return 0;
    const uint64_t d = geo_dist2(c, p.z + q.z, row, geo);
    return gauss ? geo_gaussian(d, row, table) : geo_bisquare(d, row);
}

uint64_t fx_ratio63(uint64_t num, uint64_t den) { return ratio63(num, den); }

uint64_t fx_square(uint64_t w) { return square(w); }

double fx_squares(const float* s, int n, double acc)
{
    Squares q;
    for (int i = 0; i < n; i++) q.add(s[i]);
    return acc + q.sum();
}

}
