// Which segment of which columns a warp of the residual solver's line kernel works on (solver.cu): LWARPS warps
// a block in groups of S, a group being the S segments of 32 columns. The last LWARPS % S warps have no
// group: they work on nothing, but reach the block's barriers.
#pragma once

#ifdef __CUDACC__
#define ATJUP_HD __host__ __device__ __forceinline__
#else
#define ATJUP_HD inline
#endif

namespace atjup {

constexpr int LSEG = 10, LWARPS = 8;       // levels of a segment, warps of a block

struct LineRole {
    bool on;           // the warp has a group
    int group;         // its columns' group
    int s, S;          // its segment, of S (0 of 1 without a group: no neighbour is read)
    int w0;            // the group's first warp: w0 .. w0 + S - 1 are below LWARPS
};

ATJUP_HD LineRole line_role(int w, int S) {
    LineRole r;
    r.group = w / S;
    r.on = r.group < LWARPS / S;
    r.s = r.on ? w - r.group * S : 0;
    r.S = r.on ? S : 1;
    r.w0 = w - r.s;
    return r;
}

}  // namespace atjup
