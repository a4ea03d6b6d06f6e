// Checks of pdpd_footprint.hpp, run by test_footprint.py: prints one line per failed check.
#include <cstdio>

#include "../poets-dpd_gb300/csrc/pdpd_footprint.hpp"

using namespace pdpd;

static int failed = 0;
#define CHECK(c) \
    if (!(c)) { \
        std::printf("line %d: %s\n", __LINE__, #c); \
        failed++; \
    }

static BatchSize world(int x, int y, int z, double density)
{
    const int32_t box[3] = {x, y, z};
    BatchSize s;
    s.add((uint32_t)(density * x * y * z), box, 0, 0, false);
    return s;
}

int main()
{
    // a batch of equal worlds has the buckets of one
    for (double rho : {0.01, 0.3, 1.0, 3.0, 10.0, 64.0, 200.0}) {
        BatchSize b;
        for (int k = 0; k < 5; k++) b.add(world(8, 8, 8, rho));
        CHECK(b.bucket_k() == world(8, 8, 8, rho).bucket_k());
        CHECK(b.bucket_k() % 4 == 0 && b.bucket_k() >= rho);
    }
    // mixed densities: no more bucket entries than the worlds take one by one, and so no more bytes
    const BatchSize dense = world(6, 6, 6, 30), sparse = world(100, 100, 100, 0.1), usual = world(40, 40, 40, 3);
    for (const BatchSize *x : {&dense, &sparse, &usual})
        for (const BatchSize *y : {&dense, &sparse, &usual}) {
            BatchSize b = *x;
            b.add(*y);
            CHECK(b.bucket_k() * b.cells <= x->bucket_k() * x->cells + y->bucket_k() * y->cells + 4 * b.cells * (b.bucket_k() == 4));
            for (bool fp64 : {false, true})
                if (!fp64 || (b.lists_pay() == x->lists_pay() && b.lists_pay() == y->lists_pay()))
                    CHECK(b.bytes(fp64) <= x->bytes(fp64) + y->bytes(fp64) + 1024);
        }
    // admission: within the budget; the first job at any size; FP64 not beyond the lists' reach
    const size_t GB = size_t(1) << 30;
    for (bool fp64 : {false, true}) {
        BatchSize b;
        CHECK(job_joins(b, world(400, 400, 400, 3), fp64, GB));
        uint64_t n = 0;
        for (; n < 100000 && job_joins(b, usual, fp64, 40 * GB); n++) b.add(usual);
        CHECK(n > 0 && n < 100000);
        CHECK(b.bytes(fp64) <= 40 * GB);
        CHECK(!fp64 || b.lists_fit());
        CHECK(fp64 || b.beads > (1u << 26));
        // (the snapshot buffers hold what the budget admits)
        CHECK(snapshot_reserve(fp64, 40 * GB) >= 72 * b.beads);
        CHECK(snapshot_reserve(fp64, 4 * GB) <= 72 * (4 * GB / BEAD_BYTES32));
    }
    CHECK(snapshot_reserve(true, 40 * GB) <= 72 * (size_t(1) << 25));
    // a job beyond the lists' reach runs, alone or with others
    const BatchSize giant = world(300, 300, 300, 3);
    CHECK(!giant.lists_fit() && giant.bytes(true) < 40 * GB);
    CHECK(job_joins(BatchSize{}, giant, true, GB) && job_joins(giant, usual, true, 80 * GB));
    CHECK(!job_joins(usual, giant, true, 80 * GB) && job_joins(usual, giant, false, 80 * GB));
    // a batch that takes no lists has no such limit
    const BatchSize thin = world(512, 512, 512, 0.2);
    CHECK(!thin.lists_pay() && job_joins(thin, thin, true, 200 * GB));
    return failed ? 1 : 0;
}
