// sweep_kernels.cu -- single-domain launches of the fused directional sweep
// (sweep_core.cuh): work items, TMA tensor maps and the instantiations for
// {FP64, mixed} x {plain, learned routing, guard-only routing, label
// collection}.
#include "sweep_core.cuh"

namespace how {

namespace {

// Lines per warp: four, whose rows are 32 bytes in y and z.  An x sweep takes one
// line per warp, in chunks of 32 cells, where that makes 19% less chunks of
// the domain, that is where lanes would be left without a line (1, 2, 3, 5, 6 or
// 9 lines a plane; 13 give 18.7% at best and lost 2% of a 4096 x 13 step).  FP64
// x sweep with four lines and with one:
// 1e5 cells of one line 75 and 26 us, 1024 x 1 x 1024 623 and 168, 1024 x 3 x 400
// 279 and 201, 1024 x 5 x 200 280 and 164; 96^3, where no lane is idle, 186 and 191.
constexpr int kLines = 4;
template <int NL> double line_chunks(const Grid& g) {   // of a plane, with a quarter for each line's start
    using CUT = Cut<0, NL>;
    return CUT(g, 1).groups * ((g.nx - CUT::f0) / CUT::W + 1.25);
}
int sweep_lines(const Grid& g, int dir) {
    return dir == 0 && line_chunks<1>(g) <= 0.81 * line_chunks<kLines>(g) ? 1 : kLines;
}

// Length of the work items, in chunks: the one with the least sweep_time.  Once
// no quarter of an SM gets a second item, longer ones only take longer: the
// search ends there (at 2e6 cells in one line trying every length takes 2 ms).
struct Plan { int chunks; long long each; };   // each: items per quarter of an SM
template <int DIR, int NL>
Plan pick_chunks(const Grid& g, int nsm, int warps) {
    using CUT = Cut<DIR, NL>;
    const int n = DIR == 0 ? g.nx : DIR == 1 ? g.ny : g.nz;
    const int most = (n - CUT::f0) / CUT::W + 1;
    Plan best{1, 0};
    double best_t = 0.0;
    for (int s = 1; s <= most; ++s) {
        const long long items = CUT(g, s).items(), each = (items + 4 * nsm - 1) / (4 * nsm);
        const double t = sweep_time(items, s, nsm, warps);
        if (s == 1 || t < best_t) { best = Plan{s, each}; best_t = t; }
        if (each <= 1) break;
    }
    return best;
}

template <int DIR, int NL, int WPB, typename R, int MODE>
void launch_plan(Ctx& c, SweepArgs& a, const Plan& plan) {
    constexpr int bytes = WPB * WarpMem<DIR, NL, R, MODE>::bytes + 128;
    const auto kern = k_sweep<DIR, NL, WPB, R, 1, MODE>;
    c.smem.raise((const void*)kern, bytes);
    a.seg_chunks = plan.chunks;
    // persistent grid: one block per SM (a kernel with tensor memory)
    const long long items = Cut<DIR, NL>(c.g, plan.chunks).items();
    const int grid = (int)(items < c.sm_count ? items : c.sm_count);
    cudaEvent_t ev[2];
    timer_begin(c, ev);
    kern<<<grid, 32 * WPB, bytes, c.stream>>>(a);
    timer_end(c, ev);
    ++c.launches;
}

// WPB warps per SM; SMALL (0: none) where no quarter of an SM gets more than
// SMALL / 4 items
template <int DIR, int NL, int WPB, int SMALL, typename R, int MODE>
void launch_lines(Ctx& c, SweepArgs& a) {
    const Plan plan = pick_chunks<DIR, NL>(c.g, c.sm_count, WPB / 4);
    if constexpr (SMALL > 0)
        if (plan.each <= SMALL / 4) return launch_plan<DIR, NL, SMALL, R, MODE>(c, a, plan);
    launch_plan<DIR, NL, WPB, R, MODE>(c, a, plan);
}

template <int DIR, int WPB, int SMALL, typename R, int MODE>
void launch_one(Ctx& c, SweepArgs& a) {
    if constexpr (DIR == 0)
        if (sweep_lines(c.g, DIR) == 1) return launch_lines<DIR, 1, WPB, SMALL, R, MODE>(c, a);
    launch_lines<DIR, kLines, WPB, SMALL, R, MODE>(c, a);
}

template <int DIR, int NL>
int make_maps_lines(Ctx& c) {
    using M = WarpMem<DIR, NL, double, 0>;   // the TMA boxes do not depend on R or MODE
    for (int b = 0; b < 6; ++b) {
        int rc = encode_sweep_maps(c.g, DIR, NL, M::W, M::TO, c.qbuf[b], &c.tm_in[b][DIR], &c.tm_out[b][DIR]);
        if (rc) return rc;
    }
    return 0;
}

template <int DIR>
int make_maps_dir(Ctx& c) {
    if constexpr (DIR == 0)
        if (sweep_lines(c.g, DIR) == 1) return make_maps_lines<DIR, 1>(c);
    return make_maps_lines<DIR, kLines>(c);
}

}  // namespace

// The maps of one stage buffer: the raw tile (`cells` new cells of `lines`
// lines, 8 variables) and the update operand (`op_cells`).
int encode_sweep_maps(const Grid& g, int dir, int lines, int cells, int op_cells, const double* buf, CUtensorMap* in,
                      CUtensorMap* out) {
    const uint64_t dims[4] = {(uint64_t)g.P0, (uint64_t)g.P1, (uint64_t)g.P2, 8};
    const uint64_t strides[3] = {(uint64_t)g.pitch * 8, (uint64_t)g.pitch * g.P1 * 8, (uint64_t)g.fs * 8};
    uint32_t bin[4] = {1, 1, 1, 8}, bout[4] = {1, 1, 1, 8};
    const int across = dir == 0 ? 1 : 0;
    bin[dir] = (uint32_t)cells; bin[across] = (uint32_t)lines;
    bout[dir] = (uint32_t)op_cells; bout[across] = (uint32_t)lines;
    const int rc = encode_tensor_map_4d(in, buf, dims, strides, bin);
    return rc ? rc : encode_tensor_map_4d(out, buf, dims, strides, bout);
}

int make_sweep_tensor_maps(Ctx& c) {
    int rc = make_maps_dir<0>(c);
    if (!rc) rc = make_maps_dir<1>(c);
    if (!rc) rc = make_maps_dir<2>(c);
    return rc;
}

static int buffer_of(const Ctx& c, const double* p) {
    for (int b = 0; b < 6; ++b) if (c.qbuf[b] == p) return b;
    return -1;
}

// a.qprev / a.qout / a.q0 choose the tensor maps: the tile comes from qprev;
// the update operand is q(iw) when accumulating (mode 0) or when the base was
// prepared in q(iw) (stage 5), else q(0).
void launch_sweep(Ctx& c, int dir, const SweepArgs& a_in) {
    SweepArgs a = a_in;
    a.prof = c.prof;
    a.status = &c.dsc->status;
    a.gam2 = (a.gam - 2.0) / (a.gam - 1.0);
    const int bin = buffer_of(c, a.qprev);
    const int bout = buffer_of(c, (a.mode == 0 || a.stage5) ? a.qout : a.q0);
    a.tm_in = c.tm_in[bin][dir];
    a.tm_out = c.tm_out[bout][dir];
    a.router = c.router_w;
    a.route_prev = c.route_prev ? c.route_prev + (size_t)(2 * dir + c.route_par[dir]) * c.g.fs : nullptr;
    a.route_next = c.route_prev ? c.route_prev + (size_t)(2 * dir + 1 - c.route_par[dir]) * c.g.fs : nullptr;
    a.route_count = c.route_count;
    a.collect = c.collect;
    a.collect_n = c.collect_n;
    a.collect_cap = c.collect_cap;
    a.collect_every = c.collect_every > 0 ? c.collect_every : 1;
    a.route_thr = c.route_thr;
    a.guard_jump = c.guard_jump;
    a.guard_floor = c.guard_floor;
    a.ct4 = c.p.ct_avg == 4;
    a.wait_expire = c.wait_expire;
    const bool mixed = c.precision == HOW_PREC_MIXED;
    const int mode = c.route_mode;
    if (mode == 1) {
        // learned routing: the routing pass forms fresh decisions (on the
        // stages stage_sweeps marks due) into the other half of this
        // direction's pair, which then becomes the current one; the sweep
        // reads the current decisions
        if (c.route_due) {
            launch_route(c, dir, a.qprev, a.route_prev, a.route_next);
            c.route_par[dir] ^= 1;
        }
        a.route_next = c.route_prev + (size_t)(2 * dir + c.route_par[dir]) * c.g.fs;
        a.route_prev = nullptr;
    }
    // instantiations: {fp64, mixed} x {plain, learned, guard-only}; label
    // collection runs the FP64 method.  Template arguments: warps per SM, whose
    // number caps the registers, and the warps of small domains.  FP64 at 12
    // (168 registers): 2.45 ms per 256^3 sweep, against 2.63 at 8 (250); small
    // domains at 8, whose chunk is shorter: 128^2 14.9 against 15.6 us.  Mixed at 12
    // (168 registers): 0.76 ms per 192^3 sweep, against 0.89 at 8.
#define HOW_SWEEP_CASES(D)                                                  \
    do {                                                                    \
        if (mode == 3) { launch_one<D, 8, 0, double, 3>(c, a); break; }     \
        if (mixed) {                                                        \
            if (mode == 1) launch_one<D, 12, 0, float, 1>(c, a);            \
            else if (mode == 2) launch_one<D, 12, 0, float, 2>(c, a);       \
            else launch_one<D, 12, 0, float, 0>(c, a);                      \
        } else {                                                            \
            if (mode == 1) launch_one<D, 8, 0, double, 1>(c, a);            \
            else if (mode == 2) launch_one<D, 8, 0, double, 2>(c, a);       \
            else launch_one<D, 12, 8, double, 0>(c, a);                     \
        }                                                                   \
    } while (0)
    if (dir == 0) HOW_SWEEP_CASES(0);
    else if (dir == 1) HOW_SWEEP_CASES(1);
    else HOW_SWEEP_CASES(2);
    if (mode == 2 || mode == 3) {
        // guard-only routing and label collection write the decision arrays
        c.route_par[dir] ^= 1;
        c.route_valid = false;
    }
#undef HOW_SWEEP_CASES
}

}  // namespace how
