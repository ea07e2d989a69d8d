// ReadBackPlan (2dradiation_b200/csrc/read_back_plan.hpp): every choice of up
// to 7 arrays, with chunks below, at and above an array's length.  Prints the
// first expectation that fails; exits 0 when none does.
#include <cstdio>
#include <vector>

#include "read_back_plan.hpp"

#define EXPECT(x)                                                                                         \
    do                                                                                                    \
        if (!(x))                                                                                         \
        {                                                                                                 \
            std::printf("line %d: %s (mask %d, per %d, chunk %d)\n", __LINE__, #x, mask, per, chunk);     \
            return 1;                                                                                     \
        }                                                                                                 \
    while (0)

int main()
{
    double here;
    for (int mask = 0; mask < 128; mask++)
        for (int per : {1, 5, 8})
            for (int chunk : {1, 3, 5, 7, 16, 40, 41, 1000})
            {
                double *dst[7];
                int wanted = 0;
                for (int q = 0; q < 7; q++)
                {
                    dst[q] = (mask >> q) & 1 ? &here : nullptr;
                    wanted += (mask >> q) & 1;
                }
                const grlbm::ReadBackPlan plan(dst, 7, per, chunk);
                std::vector<int> got(7 * per, 0);
                int64_t moved = 0;
                for (int64_t k = 0; k < plan.chunks(); k++)
                {
                    std::vector<int64_t> half(chunk, -1); // the source value at each place
                    plan.copies(k, [&](int64_t from, int64_t n, int64_t place) {
                        moved += n;
                        for (int64_t i = 0; i < n; i++)
                            half.at(place + i) = from + i;
                    });
                    bool right = true;
                    plan.parts(k, [&](int q, int64_t e, int64_t n, int64_t place) {
                        right = right && dst[q];
                        for (int64_t i = 0; i < n; i++)
                        {
                            right = right && half.at(place + i) == q * per + e + i;
                            got.at(q * per + e + i)++;
                        }
                    });
                    EXPECT(right);
                }
                EXPECT(moved == (int64_t)wanted * per); // what is not wanted stays on the device
                for (int q = 0; q < 7; q++)
                    for (int i = 0; i < per; i++)
                        EXPECT(got[q * per + i] == (dst[q] ? 1 : 0));
            }
    return 0;
}
