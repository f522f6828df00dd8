// certain_miss (index_math.h) against the oracle's getIndex
// (oracle/tsdf_oracle.c): wherever it says so, getIndex misses -- on maps of
// even and odd sub_dim, with and without room beyond the last brick, at
// resolutions up to and above 1 m, for offsets around every bound, NaN and
// infinities.  Prints how many points were checked and settled.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "index_math.h"
#include "map_host.h"

extern "C" {
#include "tsdf_oracle.h"
}

namespace tsdfl {
void set_error(const char*, ...) {}
}
using namespace tsdfl;

int main(int argc, char** argv)
{
    const long n = argc > 1 ? atol(argv[1]) : 200000;
    const float ress[] = {0.064f, 0.05f, 0.1f, 0.07f, 0.2f, 0.33f, 1.0f, 1.5f};
    const float sizes[][3] = {{21.3f, 17.7f, 6.1f}, {4.0f, 3.0f, 2.0f}, {0.5f, 2.2f, 1.0f}, {9.95f, 1.0f, 3.4f}};
    const float mins[][3] = {{0, 0, 0}, {-4.096f, -8.192f, -0.3f}};
    std::mt19937_64 rng(4);
    long bad = 0, checked = 0, settled = 0, misses = 0;
    for (float res : ress)
        for (auto& size : sizes)
            for (auto& mn0 : mins) {
                float mn[3] = {mn0[0], mn0[1], mn0[2]};
                float mx[3] = {mn[0] + size[0], mn[1] + size[1], mn[2] + size[2]};
                orc_map_coef c;
                orc_map_coef_init(&c, mn, mx, res, 0.0f);
                std::vector<int32_t> go(c.grid_occ_size);
                const int32_t S3 = (int32_t)(c.sub_dim * c.sub_dim_2);
                int32_t off = 0;
                for (auto& g : go) {
                    g = rng() % 6 == 0 ? -1 : off;
                    if (g >= 0) off += S3;
                }
                c.data_size = (uint64_t)off;
                tsdfl_map_coef tc;
                static_assert(sizeof(tc) == sizeof(c), "one layout");
                std::memcpy(&tc, &c, sizeof(tc));
                MapView v{};
                v.res = res;
                v.mmax_x = coarse_mmax(c.dim_x, res);
                v.mmax_y = coarse_mmax(c.dim_y, res);
                v.mmax_z = coarse_mmax(c.dim_z, res);
                auto lim = [](int32_t mm) { return mm < 0 ? 0u : bits_of((float)(mm + 1)); };
                v.lim_x = lim(v.mmax_x);
                v.lim_y = lim(v.mmax_y);
                v.lim_z = lim(v.mmax_z);
                float far[4];
                miss_bounds(tc, v.mmax_x, v.mmax_y, far);
                v.far_limit = far[0];
                v.far_x = far[1];
                v.far_y = far[2];
                v.far_z = far[3];
                std::uniform_real_distribution<float> U(-3.5f, 25.0f);
                const float special[] = {-1.0f, -0.99999994f, -1.0000001f, -0.0f, 0.0f, 0.99999994f, 1.0f, -2.0f, NAN,
                                         INFINITY, -INFINITY, 4194304.0f, -4194304.0f, 4194303.5f, -4194303.5f, 1e20f,
                                         -1e20f};
                for (long i = 0; i < n; ++i) {
                    float p[3], o[3];
                    for (int a = 0; a < 3; ++a) {
                        const uint64_t r = rng();
                        float w = U(rng);
                        if (r % 11 == 0) w = special[(r >> 8) % 17];
                        else if (r % 11 == 1) w = (float)((int)((r >> 8) % 30) - 4) + ((r >> 40) % 2 ? -1e-6f : 1e-6f);
                        else if (r % 11 == 2) w = (float)((int)((r >> 8) % 30) - 4);
                        else if (r % 11 < 6) w = std::fmod(w, size[a] + 1.0f);
                        p[a] = mn[a] + w;
                        o[a] = p[a] - mn[a];
                    }
                    ++checked;
                    const bool miss = orc_get_index(&c, go.data(), p[0], p[1], p[2]) >= c.data_size;
                    misses += miss;
                    if (!certain_miss(v, o[0], o[1], o[2])) continue;
                    ++settled;
                    if (!miss && bad++ < 10)
                        printf("res=%g sub_dim=%llu o=(%.9g %.9g %.9g): settled as a miss, is none\n", res,
                               (unsigned long long)c.sub_dim, o[0], o[1], o[2]);
                }
            }
    printf("checked %ld misses %ld settled %ld bad %ld\n", checked, misses, settled, bad);
    return bad ? 1 : 0;
}
