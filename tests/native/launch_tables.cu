// Every launch wrapper that reads a twiddle table refuses a launch without it, before
// any CUDA call.  Prints one line per call: status and the library's message.
#include <cstdio>

#include "ps_launch.cuh"

namespace ps {
PS_EXTERN_L3(float)
}
using namespace ps;

static float2 some[1];  // stands for a table that is there; no call below gets past its check

static void report(const char* what, int status) { printf("%s|%d|%s\n", what, status, ps_gpu_last_error()); }

template <int N> static void check(const char* size)
{
    using L = L3<float, N>;
    char name[64];
    const auto line = [&](const char* what, int status) {
        snprintf(name, sizeof(name), "%s@%s", what, size);
        report(name, status);
    };
    int nb = 0;
    FwdXItem<float> it{};
    it.stride = it.ncols = 16;
    ProdItem<float> pr{};
    Tables<float> t{some, some, some};
    t.twp = nullptr;
    line("inv_x", L::inv_x(0, some, 16, some, 16, LOAD_PLAIN, nullptr, 1, t));
    line("fwd_x", L::fwd_x(0, &it, 1, 16, SPEC_STORE, some, 16, nullptr, 0, t, nullptr));
    line("fwd_x sums", L::fwd_x(0, &it, 1, 16, SPEC_COUNT, nullptr, 0, nullptr, 0, t, &nb));
    if (N >= 512) t.twp = some;  // the Y pass has a table of its own there (twp_alt)
    line("pass_y", L::pass_y(0, some, 16, true, t));
    for (int q = 0; q < 2; q++) {
        t = Tables<float>{some, some, some};
        (q ? t.twr : t.twpp) = nullptr;
        line("inv_z", L::inv_z(0, some, 16, 1, nullptr, nullptr, EPI_REDUCE, 1, nullptr, t, &nb));
        line("fwd_z", L::fwd_z(0, SRC_F32, some, nullptr, some, 16, 1, t));
        line("pair_z", L::pair_z(0, some, 16, 1, some, 16, 1, some, 16, 1, t));
        line("prod_z", L::prod_z(0, &pr, 1, 1, false, 0, t, &nb));
    }
}

int main()
{
    check<64>("64");
    check<384>("384");
    check<512>("512");
    check<1024>("1024");
    return 0;
}
