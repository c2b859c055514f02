// Planning of resident collider solves, shared by the single-domain entry
// points and the batched plan (definitions in ffx_graph_resident.cu).
#pragma once
#include <vector>

#include "ffx_graph_resident.cuh"

namespace ffx {
namespace gres {

constexpr int kHeader = 160;       // words: two exchange numbers per block, the timeout count last

// A domain's hierarchy. whole: level 0 is the mask's grid.
struct Spec {
    int count;
    bool whole;
    const double* inverse;
    int pre0, post0, pre, post, last;
    float omega;
    FfxGraphLevel level[kLevels];
};

// Tiles of ty x tz rows on level 0; blocks counts the tail's.
struct Candidate {
    int ty, tz, blocks;
    double cost;
};

// Tiles for every domain so that all blocks of all domains are resident on `sms`
// SMs at once; false when they do not fit. dist: levels in tiles, per domain.
bool plan_blocks(const Spec* specs, int count, int sms, std::vector<Candidate>& chosen, std::vector<int>& dist);
// 64-bit words of a domain's published rows and header.
int64_t words_of(const Spec& S, int dist);
// The domain's record; returns the bytes of shared memory its blocks need.
int fill(const Spec& S, int dist, const Candidate& c, int first_block, u64* ws, Domain& D);
int launch(bool links, const Domain* domains, int count, int blocks, int smem, const Call& A, cudaStream_t st);

}  // namespace gres
}  // namespace ffx
