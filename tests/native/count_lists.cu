// The lists of exact polygon counts on the host: modes of interval shells from their
// orbits against a walk over the whole grid, and which pairs of shells are listed.
#include <cstdio>
#include <set>
#include <tuple>

#include "ps_counts.cuh"
using namespace ps;

static Shell shell(int lo, int hi, int band)
{
    Shell s{};
    s.kind = SHELL_RANGE;
    s.r2lo = lo;
    s.r2hi = hi;
    s.band = band;
    return s;
}
static Shell thick(double r, double w, int n)
{
    const double lo = r - w / 2, hi = r + w / 2;
    return shell(lo > 0 ? (int)std::ceil(lo * lo) : 0, (int)std::floor(hi * hi), std::min((int)hi, n / 2));
}

static int check(const Shell& s, int n)
{
    std::set<std::tuple<int, int, int>> want, got;
    const int b = std::min(s.band, n / 2);
    for (int x = -n / 2; x < n / 2; x++)
        for (int y = -n / 2; y < n / 2; y++)
            for (int z = -n / 2; z < n / 2; z++) {
                const int r2 = x * x + y * y + z * z;
                if (std::max({std::abs(x), std::abs(y), std::abs(z)}) <= b && r2 >= s.r2lo && r2 <= s.r2hi)
                    want.insert({x, y, z});
            }
    const std::vector<int4> reps = interval_orbits(s, n);
    const std::vector<short4> modes = orbit_modes(reps, n);
    for (const short4& m : modes) got.insert({m.x, m.y, m.z});
    return modes.size() == want.size() && orbit_total(reps) == want.size() && got == want;
}

int main()
{
    int bad = 0, done = 0;
    for (int n : {16, 24, 30, 48})
        for (int hi : {0, 1, 2, 3, 5, 9, 27, 48, 75, 64, 100, 192, n * n / 4, n * n / 4 + 7, n * n / 2, 3 * n * n / 4})
            for (int w : {0, 1, 4, 40, 5000}) {
                const int band = std::min(n / 2, (int)std::sqrt((double)hi));
                bad += !check(shell(std::max(0, hi - w), hi, band), n);
                done++;
            }
    bad += !check(shell(5, 4, 2), 16) + !check(shell(0, -1, 0), 16);
    printf("modes %d of %d wrong\n", bad, done + 2);
    // sides (in grid points), thickness, transforms' grid: enumerated or not
    struct { int n, m; double r, w; int one, want; } rule[] = {
        {128, 128, 60.0, 1.0, 1, 1},    // thin triangles of a 128^3 list
        {128, 128, 57.6, 6.4, 1, 0},    // the same, thick: 1.6e9 pairs, more than the transforms cost
        {256, 256, 70.0, 12.8, 1, 0},   {256, 256, 60.0, 1.0, 1, 1}, {512, 384, 80.0, 1.0, 1, 1},
        {512, 512, 230.0, 1.0, 1, 0},   {600, 320, 100.0, 1.0, 1, 1}, {600, 600, 270.0, 1.0, 1, 0},
        {512, 384, 90.0, 1.0, 0, 1},    {512, 384, 90.0, 20.0, 0, 0},
    };
    for (const auto& q : rule) {
        PairCountLists L;
        const Shell s = thick(q.r, q.w, q.n);
        const bool got = pair_count_lists(s, s, q.n, q.m, 0, 0x7fffffff, q.one != 0, &L);
        const double pairs = (double)L.reps.size() * (double)orbit_total(L.reps);
        printf("rule n %d m %d r %.1f w %.1f one %d: %d want %d, reps %zu, pairs %.2e, modes %zu\n", q.n, q.m, q.r, q.w,
               q.one, (int)got, q.want, L.reps.size(), pairs, L.modes.size());
    }
    return 0;
}
