// Host check of DgStore::poison (hsr_digits.cuh): a product cut into parts of
// its inner columns marks every entry of every part, and nothing beside them.
// Prints "<entries not marked> <others marked>".
#include <cmath>
#include <cstdio>
#include <vector>

#include "../../hsrq3in_gb300/csrc/hsr_digits.cuh"

using namespace hsr;

int main() {
    int missed = 0, beside = 0;
    for (const int steps : {1, 8, 23})
        for (const int per : {1, 5, 8, 23}) {
            const int M = 130, N = 7, ld = M + 3, parts = (steps + per - 1) / per;
            const long long cz = (long long)ld * N + 11;
            std::vector<double> out((size_t)(cz * (parts + 1)), 1.0);
            DgStoreLong e{2, 1, steps, per, M, N, nullptr, nullptr, out.data(), 1, ld, cz};
            for (int t = 0; t < 64; ++t) e.poison(t, 64);
            for (long long q = 0; q < (long long)out.size(); ++q) {
                const long long z = q / cz, r = q % cz;
                const bool in = z < parts && r / ld < N && r % ld < M;
                if (in && !std::isnan(out[(size_t)q])) ++missed;
                if (!in && std::isnan(out[(size_t)q])) ++beside;
            }
        }
    std::printf("%d %d\n", missed, beside);
    return missed != 0 || beside != 0;
}
