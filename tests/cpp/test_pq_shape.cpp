// The rows and shapes that the tensor-core product-quantizer kernel is given, on the host.
#include <climits>
#include <cstdio>

#include "../../vq_b200/csrc/pq_tc_shape.hpp"

#define CHECK(c)                                              \
    do {                                                      \
        if (!(c)) return std::printf("%s: failed\n", #c), 1; \
    } while (0)

int main()
{
    using namespace vqb;
    const size_t limit = size_t(1) << 31;
    CHECK(!pq_tc_rows(0) && pq_tc_rows(1) && pq_tc_rows(limit - 1) && pq_tc_rows(limit));
    CHECK(!pq_tc_rows(limit + 1) && !pq_tc_rows(limit + PQ_TC_TILE) && !pq_tc_rows((size_t(1) << 32) - 1) && !pq_tc_rows(size_t(1) << 32));
    // the first row of every tile of a call is a coordinate that TMA can be given
    CHECK((limit - 1) / PQ_TC_TILE * PQ_TC_TILE <= (size_t)INT_MAX);
    CHECK(pq_tc_shape(4, 4, 2) && pq_tc_shape(64, 8, 256) && pq_tc_shape(7, 8, 100));
    CHECK(!pq_tc_shape(3, 8, 16) && !pq_tc_shape(65, 8, 16) && !pq_tc_shape(8, 16, 16) && !pq_tc_shape(8, 8, 1) && !pq_tc_shape(8, 8, 257));
    return 0;
}
