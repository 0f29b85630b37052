// ensemble_sweep.cu -- the fused sweep over every member of a batched
// ensemble in one persistent launch, for each work-item shape the autotuner
// may pick.  Member m's items occupy [tile_start[m], tile_start[m+1]) of the
// launch's item space; each item reads its member's arguments (geometry,
// stage pointers, TMA tensor maps, dt) from a device table.
#include "sweep_core.cuh"
#include "ensemble.cuh"

namespace how {

namespace {

// Candidate shapes per direction: lines per warp and chunks per work item
// (k_sweep).  Short items spread small members over the chip, long ones repeat
// less work at segment ends; one line per warp suits 1-D members.  y/z lines
// are consecutive i and NL is even there (16-byte TMA rule).
struct ShapeDef { int nl, chunks; };
constexpr ShapeDef kShapes[3][kEnsShapes] = {
    {{4, 2}, {4, 8}, {1, 2}},
    {{4, 2}, {4, 8}, {2, 2}},
    {{4, 2}, {4, 8}, {4, 4}},
};
constexpr int kWarps = 12, kBlocks = 1;   // warps per block, blocks per SM: as the single-domain FP64 sweep

template <int DIR, int NL>
void launch_ens(SweepArgs a0, int chunks, cudaStream_t st, int blocks, SmemLimits& smem) {
    constexpr int bytes = kWarps * WarpMem<DIR, NL, double, 0>::bytes + 128;
    const auto kern = k_sweep<DIR, NL, kWarps, double, kBlocks, 0, true>;
    smem.raise((const void*)kern, bytes);
    a0.seg_chunks = chunks;
    kern<<<blocks, 32 * kWarps, bytes, st>>>(a0);
}

template <int DIR>
long long items_of(const Grid& g, int nl, int chunks) {
    switch (nl) {
        case 1: return Cut<DIR, 1>(g, chunks).items();
        case 2: return Cut<DIR, 2>(g, chunks).items();
        default: return Cut<DIR, 4>(g, chunks).items();
    }
}

}  // namespace

// (lines, cells a work item advances along the sweep)
void ens_shape(int dir, int s, int* nl, int* t) {
    const ShapeDef& d = kShapes[dir][s];
    *nl = d.nl;
    *t = d.chunks * (32 / d.nl) - (dir == 0 ? 2 : 1);
}

int ens_chunks(int dir, int s) { return kShapes[dir][s].chunks; }
int ens_line_chunks(const Grid& g, int dir, int s) {
    const int w = 32 / kShapes[dir][s].nl;
    return dir == 0 ? (g.nx + 1) / w + 1 : (dir == 1 ? g.ny : g.nz) / w + 1;   // (x: from interface -1)
}

long long ens_tiles(const Grid& g, int dir, int s, int chunks) {
    const int n = dir == 0 ? g.nx : dir == 1 ? g.ny : g.nz;
    if (n <= 1) return 0;
    const int nl = kShapes[dir][s].nl;
    return dir == 0 ? items_of<0>(g, nl, chunks) : dir == 1 ? items_of<1>(g, nl, chunks) : items_of<2>(g, nl, chunks);
}

// Tensor maps of the 6 stage buffers of a context for shape s of direction dir.
int ens_encode_maps(const Ctx& c, int dir, int s, CUtensorMap* tm_in, CUtensorMap* tm_out) {
    const int nl = kShapes[dir][s].nl, w = 32 / nl;
    for (int b = 0; b < 6; ++b) {
        const int rc = encode_sweep_maps(c.g, dir, nl, w, dir == 0 ? w + 2 : w, c.qbuf[b], &tm_in[b], &tm_out[b]);
        if (rc) return rc;
    }
    return 0;
}

void ens_launch_sweep(int dir, int s, int chunks, long long items, const SweepArgs& a0, cudaStream_t st, int nsm,
                      SmemLimits& smem) {
    const ShapeDef& d = kShapes[dir][s];
    const int blocks = (int)(items < nsm ? items : nsm);   // one per SM
    if (dir == 0) {
        if (d.nl == 1) launch_ens<0, 1>(a0, chunks, st, blocks, smem);
        else launch_ens<0, 4>(a0, chunks, st, blocks, smem);
    } else if (dir == 1) {
        if (d.nl == 2) launch_ens<1, 2>(a0, chunks, st, blocks, smem);
        else launch_ens<1, 4>(a0, chunks, st, blocks, smem);
    } else {
        launch_ens<2, 4>(a0, chunks, st, blocks, smem);
    }
}

}  // namespace how
