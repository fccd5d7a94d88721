// Wall words (WALL_* in lbm_common.cuh): from the flags, and as the sweeps ask for them.
#pragma once
#include "lbm_common.cuh"

namespace lbm {

// Wall word of a near-wall fluid cell from the flags (which point at the cell; the other arguments are the
// flag field's neighbour offsets).  All loads are independent of one another.  Out of line: one copy per
// translation unit, and none of its registers in the sweeps.
template <int Q>
__device__ __noinline__ uint32_t wall_links(const uint8_t* flags, int dx0, int dx2, int dy0, int dy2, int dz0,
                                            int dz2) {
    using L = Lat<Q>;
    NbrOffsets fo;
    fo.dx[0] = dx0; fo.dx[1] = 0; fo.dx[2] = dx2;
    fo.dy[0] = dy0; fo.dy[1] = 0; fo.dy[2] = dy2;
    fo.dz[0] = dz0; fo.dz[1] = 0; fo.dz[2] = dz2;
    uint32_t w = 0;
    unsigned types = 0;
#pragma unroll
    for (int i = 1; i < Q; ++i) {
        const int t = flags[fo.off(-L::cx(i), -L::cy(i), -L::cz(i))] & FLAG_TYPE_MASK;
        types |= 1u << t;
        w |= uint32_t(t == FLAG_NOSLIP || flag_is_ubb(t)) << i;
    }
    return w | wall_kinds(types);
}

__device__ __forceinline__ NbrOffsets flag_offsets(const Grid& g, int x, int y, int z) {
    NbrOffsets fo;
    Grid gf = g;
    gf.sy = g.fsy;
    gf.sz = g.fsz;
    fo.init(gf, x, y, z);
    return fo;
}

// Wall word of any interior cell from the finalized flags.
template <int Q>
__device__ __forceinline__ uint32_t wall_word_of_flags(const Grid& g, int x, int y, int z) {
    const uint8_t* cell = g.flags + ((x + 1) + (y + 1) * g.fsy + (z + 1) * g.fsz);
    const int fl = *cell;
    if (fl & FLAG_TYPE_MASK) return WALL_SELF;
    if (!(fl & FLAG_NEAR_WALL)) return 0;
    const NbrOffsets fo = flag_offsets(g, x, y, z);
    return wall_links<Q>(cell, fo.dx[0], fo.dx[2], fo.dy[0], fo.dy[2], fo.dz[0], fo.dz[2]);
}

#ifdef __CUDACC__
// Wall word of an interior cell in two parts, with the loads of its populations between them: begin()
// asks whether the cell's row has walls at all, word() reads the cell's word if so.  A cell in another
// row, as almost all are, then waits for its populations alone, where the row's answer used to come
// first.  Without wall words begin() takes them from the flags.
template <int Q> struct WallProbe {
    uint32_t from_flags = 0;
    bool flagged = false;
    __device__ __forceinline__ void begin(const Grid& g, int x, int y, int z) {
        if (g.flags == nullptr) return;
        if (g.walls != nullptr) {
            flagged = row_flagged(g, y, z);
            return;
        }
        if (row_flagged(g, y, z)) from_flags = wall_word_of_flags<Q>(g, x, y, z);
    }
    __device__ __forceinline__ uint32_t word(const Grid& g, int x, int y, int z) const {
        return flagged ? g.walls[unsigned(x) + unsigned(g.nx) * (unsigned(y) + unsigned(g.ny) * unsigned(z))]
                       : from_flags;
    }
};

template <int Q>
__device__ __forceinline__ uint32_t wall_word(const Grid& g, int x, int y, int z) {
    WallProbe<Q> probe;
    probe.begin(g, x, y, z);
    return probe.word(g, x, y, z);
}
#endif

}  // namespace lbm
