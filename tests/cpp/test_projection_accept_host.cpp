// Host build of the test that leaves a 12 x 12 double matrix as it is (project_pd.cuh, classify12).
// Usage: test_projection_accept_host <in> <out>
//   in : int64 count, count * 144 doubles (row-major matrices)
//   out: count int32, the class of each (row-major storage), then of each in block-major storage.
#include <cmath>
#include <cstdint>
#include <fstream>
#include <vector>

#define SYMXG_DEVICE inline
static inline float rsqrtf(float x) { return 1.0f / std::sqrt(x); }
static inline float __frcp_rn(float x) { return 1.0f / x; }
using std::fabs;
using std::fmax;
using std::sqrt;
#include "../../symx_gb300/csrc/project_pd.cuh"

int main(int argc, char** argv)
{
    if (argc != 3) return 2;
    std::ifstream f(argv[1], std::ios::binary);
    int64_t count = 0;
    f.read(reinterpret_cast<char*>(&count), sizeof count);
    std::vector<double> in((size_t)count * 144);
    f.read(reinterpret_cast<char*>(in.data()), in.size() * sizeof(double));
    std::vector<int32_t> out(2 * count);
    for (int64_t e = 0; e < count; ++e) {
        const double* h = in.data() + e * 144;
        double bm[144];
        for (int i = 0; i < 12; ++i)
            for (int j = 0; j < 12; ++j) bm[symxg_dev::bm_index<12>(i, j)] = h[12 * i + j];
        out[e] = symxg_dev::classify12<true>(h, 0.0);
        out[count + e] = symxg_dev::classify12<false>(bm, 0.0);
    }
    std::ofstream g(argv[2], std::ios::binary);
    g.write(reinterpret_cast<const char*>(out.data()), out.size() * sizeof(int32_t));
    return 0;
}
