// eu3d_kernels_impl.cuh — launchers for one arithmetic flavour. Included once
// by eu3d_kernels_strict.cu (--fmad=false, exact forms) and once by
// eu3d_kernels_fast.cu, with EU3D_NS naming the namespace.
#pragma once

#include <algorithm>

#include "eu3d_attr.hpp"
#include "eu3d_kernels.cuh"
#include "eu3d_launch.hpp"

namespace eu3d {
namespace EU3D_NS {

namespace {

template <int NS, int NR>
cudaError_t boundary_t(const LaunchArgs &a)
{
    const DevGrid &g = a.g;
    // a thread per ghost node; on a grid bc nodes thick one per pair of z ghosts
    const long long n = 2LL * g.bc * ((long long)g.nj * g.nk + (long long)g.ni * g.nk) +
                        (g.nk == g.bc ? 1LL : 2LL) * g.bc * g.ni * g.nj;
    const int threads = 256;
    const long long blocks = (n + threads - 1) / threads;
    k_boundary<NS><<<dim3((unsigned)blocks), threads, 0, a.stream>>>(*a.mech, g, a.st);
    return cudaGetLastError();
}

// FP64 reconstruction: the reference's divisions (EU_EXACT_FLUX=1) or the
// division-light limiter form.
constexpr bool kStrictFlux = EU_EXACT_FLUX != 0;

inline int tiles_j(const DevGrid &g) { return (g.nj + kTileJ - 1) / kTileJ; }
inline int tiles_k(const DevGrid &g) { return (g.nk + kTileK - 1) / kTileK; }

// The tiled kernel's march where the autotuner has not chosen one. A block costs
// its ci planes and about three more (the window's first planes and the first
// face), and runs among two per SM: the ci whose rounds of blocks cost least
// (256 x 128 x 128: 24, 0.436 ms against 0.459 at 16; 192 x 96 x 96: 29, 0.193
// against 0.213). In a batch the rounds mix with the other instances' and the march
// counts for little: eight instances, 50 steps, 99.7 / 99.2 / 98.7 ms at 16 / 24 / 32.
inline int tiled_march(const LaunchArgs &a)
{
    const long long tiles = (long long)tiles_j(a.g) * tiles_k(a.g);
    if (a.batch_cells > 0)
        return 24;
    const long long slots = 2LL * (a.sms > 0 ? a.sms : 148);
    int best = 16;
    long long least = -1;
    for (int ci = 8; ci <= 48; ++ci) {
        const long long blocks = tiles * ((a.g.ni + ci - 1) / ci);
        const long long cost = (blocks + slots - 1) / slots * (ci + 3);
        if (least < 0 || cost < least) {
            least = cost;
            best = ci;
        }
    }
    return best;
}

inline int tiled_ci(const LaunchArgs &a)
{
    return std::max(a.tiled_ci > 0 ? a.tiled_ci : tiled_march(a), (a.g.ni + 65534) / 65535); // gridDim.z < 2^16
}

template <int NS>
cudaError_t tiled_flux_launch(const LaunchArgs &a)
{
    const DevGrid &g = a.g;
    const size_t smem = tiled_flux_smem_bytes<NS>();
    static SmemLimit limit; // per instantiation, per device
    const cudaError_t e = limit.ensure(k_flux_update_tiled<NS>, smem);
    if (e != cudaSuccess)
        return e;
    const dim3 block(kTileK, kTileWarps);
    const int ci = tiled_ci(a);
    const dim3 grid(tiles_k(g), tiles_j(g), (g.ni + ci - 1) / ci);
    k_flux_update_tiled<NS><<<grid, block, smem, a.stream>>>(g, a.st, a.st.prim32, a.dt_dev, ci);
    return cudaGetLastError();
}

// n cut into pieces of about `want`, all but the last equally long (129 at 8:
// 17 pieces of 8, the last of 1; 65 at 16: five of 13).
inline int even_piece(int n, int want)
{
    const int pieces = (n + want - 1) / want;
    return (n + pieces - 1) / pieces;
}

// Grids of few cells leave SMs without blocks when the tiles hold 128 of them
// (fewer than 8 blocks of 128 cells per SM): there a tile holds half the cells and
// the block twice the threads, so that a step is one round of faces a block (33 x 17
// x 17 strict: 0.023 ms against 0.033-0.054 with the large grids' tiles; 129 x 65 x 65
// FP64 the other way: 0.133 against 0.145). In a batch the cells of all instances
// count: 8 mixed ones of 44^3 take 0.154 ms a step, 0.246 with the small grids' tiles;
// 16 of 32^3 in FP64 0.238 against 0.283 (fast), 0.519 against 0.582 (strict).
inline bool small_grid(const LaunchArgs &a)
{
    return std::max((long long)a.g.ni * a.g.nj * a.g.nk, a.batch_cells) < (a.sms > 0 ? a.sms : 148) * 8LL * 128;
}

// The tile of k_flux_update_faces for a grid: 128 (small grids: 64) cells, rows
// along z cut evenly into about 8 FP64 or 16 FP32 values (the whole of a thin
// grid), 4 of them (16 on thin grids of many cells) along y, the rest along x.
template <typename R>
FaceTile face_tile(const LaunchArgs &a)
{
    const DevGrid &g = a.g;
    const bool small = small_grid(a);
    const int cells = small ? 64 : 128;
    FaceTile t;
    t.tk = even_piece(g.nk, sizeof(R) == 8 ? 8 : 16);
    t.tj = even_piece(g.nj, t.tk <= 3 && !small ? 16 : 4);
    t.ti = std::min(g.ni, std::max(1, cells / (t.tj * t.tk)));
    while (t.ti > 1 && (t.ti + 1) * t.tj * t.tk + t.ti * (t.tj + 1) * t.tk + t.ti * t.tj * (t.tk + 1) > kFacePitch<R>)
        --t.ti;
    t.y_first = (g.nj + t.tj - 1) / t.tj > 65535; // gridDim.y < 2^16
    t.d_tk = make_fastdiv(unsigned(t.tk));
    t.d_tk1 = make_fastdiv(unsigned(t.tk + 1));
    t.d_area = make_fastdiv(unsigned(t.tj * t.tk));
    t.d_area_y = make_fastdiv(unsigned((t.tj + 1) * t.tk));
    t.d_area_z = make_fastdiv(unsigned(t.tj * (t.tk + 1)));
    return t;
}

template <int NS, typename R, bool kStrict>
cudaError_t faces_flux_launch(const LaunchArgs &a, const R *prim)
{
    const DevGrid &g = a.g;
    constexpr size_t smem = face_smem_bytes<NS, R>();
    static SmemLimit limit; // per instantiation, per device
    const cudaError_t e = limit.ensure(k_flux_update_faces<NS, R, kStrict>, smem);
    if (e != cudaSuccess)
        return e;
    const FaceTile t = face_tile<R>(a);
    const int ci = std::max(std::max(a.face_ci, t.ti), (g.ni + 65534) / 65535); // gridDim.z < 2^16
    const int threads = small_grid(a) ? kFaceThreadsWide : kFaceThreads;
    const unsigned tiles_z = unsigned((g.nk + t.tk - 1) / t.tk), tiles_y = unsigned((g.nj + t.tj - 1) / t.tj);
    const dim3 grid(t.y_first ? tiles_y : tiles_z, t.y_first ? tiles_z : tiles_y, unsigned((g.ni + ci - 1) / ci));
    k_flux_update_faces<NS, R, kStrict><<<grid, threads, smem, a.stream>>>(g, a.st, prim, a.dt_dev, t, ci);
    return cudaGetLastError();
}

// The kernel of FP32 fluxes (mixed precision, always the division-light forms); the
// two give the same bits. FP64 fluxes (the reference's forms when strict, the
// division-light limiter when fast) are always formed a face a thread.
// The tiled kernel reads each primitive once but wants its 32-lane rows in z, its 7 x
// 32 tiles full and the chip filled by its blocks of eight warps. Flux of a grid
// alone, ms, tiled against faces (share of the tiles' cells that are the grid's):
//   96 x 48 x 48    0.050 0.037 (73 %)    200 x 100 x 100  0.242 0.297 (74 %)
//   100 x 50 x 50   0.051 0.048 (70 %)    129 x 65 x 65    0.089 0.094 (65 %)
//   112 x 56 x 56   0.052 0.058 (88 %)    200 x 100 x 40   0.123 0.127 (60 %)
//   128 x 64 x 64   0.064 0.077 (91 %)    256 x 128 x 33   0.189 0.171 (51 %)
//   256 x 128 x 128 0.404 0.543 (96 %)    200 x 100 x 17   0.062 0.059 (51 %)
// so it takes grids of 300,000 cells and more at 55 % and more. The instances of a
// batch share the chip: there the faces' shorter blocks are ahead up to about a
// million cells in all and the tiles beyond, down to half full (a step, ms):
//   2 x 64^3 0.129 0.103   6 x 44^3 0.147 0.112   4 x (96 x 48 x 48) 0.180 0.176
//   4 x 64^3 0.195 0.206  16 x 44^3 0.283 0.321   8 x (96 x 48 x 48) 0.322 0.360
//   8 x (64 x 33 x 33) 0.158 0.143, 16 of them 0.267 0.298 (49 %)
constexpr int kThinNk = 16;

inline bool takes_tiled(const LaunchArgs &a)
{
    const DevGrid &g = a.g;
    const bool batch = a.batch_cells > 0;
    const long long cells = batch ? a.batch_cells : (long long)g.ni * g.nj * g.nk;
    const long long slots = (long long)tiles_j(g) * kTileJ * (tiles_k(g) * kTileK);
    return g.nk >= kThinNk && cells >= (batch ? 1000000 : 300000) &&
           100LL * g.nj * g.nk >= (batch ? 45 : 55) * slots;
}

template <int NS, int NR>
cudaError_t flux_t(const LaunchArgs &a)
{
#ifdef EU_MIXED
    return takes_tiled(a) ? tiled_flux_launch<NS>(a) : faces_flux_launch<NS, float, false>(a, a.st.prim32);
#else
    return faces_flux_launch<NS, double, kStrictFlux>(a, a.st.prim);
#endif
}

template <int NS, int NR>
cudaError_t react_t(const LaunchArgs &a, bool react)
{
    const DevGrid &g = a.g;
    const long long n = (long long)g.ni * g.nj * g.nk;
    const int threads = a.recover_block > 0 ? a.recover_block : 128;
    const long long blocks = (n + threads - 1) / threads;
    const dim3 grid((unsigned)blocks);
    if (!react)
        k_recover_react<NS, NR, false, TableRates<NS, NR>><<<grid, threads, 0, a.stream>>>(*a.mech, g, a.st, a.dt_dev,
                                                                                           a.max_substeps);
    else if (a.spec == 1 && NS == Mech_JA919::NS && NR == Mech_JA919::NR) {
        // Register target, 2, 3 or 4 resident blocks per SM (autotuned, or by the
        // grid): once the cells fill two blocks a SM, more warps pay for the spills
        // (129 x 65 x 65 fast: 0.253 / 0.199 / 0.189 ms; 281 x 141 x 2 strict: 0.129 /
        // 0.095 / 0.102); below, a cell's own chain counts (33 x 17 x 17 strict: 0.041 /
        // 0.043 / 0.043).
#ifdef EU_EXACT_RATES
        constexpr int kFull = 3;
#else
        constexpr int kFull = 4;
#endif
        const bool full = n > 256LL * (a.sms > 0 ? a.sms : 148);
        const int minb = a.recover_minb > 0 ? a.recover_minb : full ? kFull : 2;
        if (minb == 4)
            k_recover_react<NS, NR, true, Mech_JA919, 4><<<grid, threads, 0, a.stream>>>(*a.mech, g, a.st, a.dt_dev,
                                                                                       a.max_substeps);
        else if (minb == 3)
            k_recover_react<NS, NR, true, Mech_JA919, 3><<<grid, threads, 0, a.stream>>>(*a.mech, g, a.st, a.dt_dev,
                                                                                       a.max_substeps);
        else
            k_recover_react<NS, NR, true, Mech_JA919, 2><<<grid, threads, 0, a.stream>>>(*a.mech, g, a.st, a.dt_dev,
                                                                                       a.max_substeps);
    } else
        k_recover_react<NS, NR, true, TableRates<NS, NR>><<<grid, threads, 0, a.stream>>>(*a.mech, g, a.st, a.dt_dev,
                                                                                          a.max_substeps);
    return cudaGetLastError();
}

template <int NS, int NR>
cudaError_t derived_t(const LaunchArgs &a, int which, double *out)
{
    const int threads = 256;
    const long long blocks = (a.g.n3 + threads - 1) / threads;
    k_derived<NS><<<dim3((unsigned)blocks), threads, 0, a.stream>>>(*a.mech, a.g, a.st, which, out);
    return cudaGetLastError();
}

template <int NS, int NR>
cudaError_t materialize_t(const LaunchArgs &a)
{
    if (!a.st.prim32)
        return cudaSuccess;
    k_materialize<NS><<<dim3(unsigned((a.g.n3 + 127) / 128)), 128, 0, a.stream>>>(*a.mech, a.g, a.st);
    return cudaGetLastError();
}

template <int NS, int NR>
cudaError_t classify_t(const LaunchArgs &a, const LearnedParams &lp)
{
    const long long n = (long long)a.g.ni * a.g.nj * a.g.nk;
    // (64 threads: 0.206 ms on 256 x 128 x 128 against 0.211 with 128)
    const int threads = a.recover_block > 0 ? a.recover_block : 64;
    const dim3 grid(unsigned((n + threads - 1) / threads));
    switch (a.recover_minb) {
    case 3: k_recover_classify<NS, 3><<<grid, threads, 0, a.stream>>>(*a.mech, a.g, a.st, lp); break;
    case 5: k_recover_classify<NS, 5><<<grid, threads, 0, a.stream>>>(*a.mech, a.g, a.st, lp); break;
    case 6: k_recover_classify<NS, 6><<<grid, threads, 0, a.stream>>>(*a.mech, a.g, a.st, lp); break;
    default: k_recover_classify<NS, 4><<<grid, threads, 0, a.stream>>>(*a.mech, a.g, a.st, lp); break;
    }
    return cudaGetLastError();
}

// The learned-chemistry kernels run on fixed grids that read the queue lengths
// on the device, so a step needs no host-side count and can be captured.
inline unsigned queue_grid(const LaunchArgs &a, int per_sm) { return unsigned((a.sms > 0 ? a.sms : 148) * per_sm); }

template <int NS, int NR>
cudaError_t apply_t(const LaunchArgs &a, const LearnedParams &lp)
{
    k_learned_apply<NS><<<dim3(queue_grid(a, 8)), 128, 0, a.stream>>>(*a.mech, a.g, a.st, lp);
    return cudaGetLastError();
}

// count[0]: queue length, count[1]: cells taken so far (zero at launch)
template <int NS, int NR>
cudaError_t react_queue_t(const LaunchArgs &a, const int *queue, int *count, int counter)
{
    const dim3 grid(queue_grid(a, 4));
    if (a.spec == 1 && NS == Mech_JA919::NS && NR == Mech_JA919::NR)
        k_react_queue<NS, Mech_JA919><<<grid, 128, 0, a.stream>>>(*a.mech, a.g, a.st, queue, count, a.dt_dev,
                                                                  a.max_substeps, counter);
    else
        k_react_queue<NS, TableRates<NS, NR>><<<grid, 128, 0, a.stream>>>(*a.mech, a.g, a.st, queue, count,
                                                                          a.dt_dev, a.max_substeps, counter);
    return cudaGetLastError();
}

template <int NS, int NR>
cudaError_t route_t(const LaunchArgs &a, const LearnedParams &lp)
{
    const dim3 grid(queue_grid(a, 4));
    if (a.spec == 1 && NS == Mech_JA919::NS && NR == Mech_JA919::NR)
        k_learned_route<NS, Mech_JA919><<<grid, 128, 0, a.stream>>>(*a.mech, a.g, a.st, lp, a.dt_dev, a.max_substeps);
    else
        k_learned_route<NS, TableRates<NS, NR>><<<grid, 128, 0, a.stream>>>(*a.mech, a.g, a.st, lp, a.dt_dev,
                                                                            a.max_substeps);
    return cudaGetLastError();
}

template <int NS, int NR>
cudaError_t state_from_tpy_t(const LaunchArgs &a, long long n, const double *T, const double *p, const double *Y,
                             double *cs, double *E)
{
    if (n <= 0)
        return cudaSuccess;
    k_state_from_tpy<NS><<<dim3(unsigned((n + 127) / 128)), 128, 0, a.stream>>>(*a.mech, n, T, p, Y, cs, E);
    return cudaGetLastError();
}

#ifdef EU_EXACT_RATES // the chemistry samples run in the strict flavour alone
template <int NS, int NR>
cudaError_t chem_samples_t(const LaunchArgs &a, long long n, double *cs, double *T, double *E, const double *dt,
                           int *nchem, int *heavy)
{
    if (n <= 0)
        return cudaSuccess;
    const dim3 grid(unsigned((n + 127) / 128));
    if (a.spec == 1 && NS == Mech_JA919::NS && NR == Mech_JA919::NR)
        k_chem_samples<NS, Mech_JA919><<<grid, 128, 0, a.stream>>>(*a.mech, n, cs, T, E, dt, nchem, a.max_substeps,
                                                                   a.st.counters, heavy);
    else
        k_chem_samples<NS, TableRates<NS, NR>><<<grid, 128, 0, a.stream>>>(*a.mech, n, cs, T, E, dt, nchem,
                                                                           a.max_substeps, a.st.counters, heavy);
    if (heavy) // one warp a deferred sample, at most a warp for each
        k_chem_heavy<NS, NR><<<dim3(unsigned(std::min<long long>((n + 3) / 4, queue_grid(a, kHeavyBlocksPerSm)))), 128,
                               0, a.stream>>>(*a.mech, n, cs, T, E, dt, nchem, a.max_substeps, a.st.counters, heavy);
    return cudaGetLastError();
}
#endif

template <int NS, int NR>
cudaError_t heavy_t(const LaunchArgs &a, int blocks)
{
    k_react_heavy<NS, NR><<<dim3(unsigned(blocks)), 128, 0, a.stream>>>(*a.mech, a.g, a.st, a.dt_dev,
                                                                         a.max_substeps);
    return cudaGetLastError();
}

// The batch's shared kinetics stage: the stiff-fallback queues, then the
// deferred cells, of every instance in tab[0..n) drained by one fixed grid
// each (next[0] and next[1] zero at launch). a: any member's arguments (the
// mechanism, flavour and substep cap are the same over the table).
template <int NS, int NR>
cudaError_t react_queue_batch_t(const LaunchArgs &a, const BatchCell *tab, int n, int *next, int counter)
{
    const dim3 grid(queue_grid(a, 4));
    if (a.spec == 1 && NS == Mech_JA919::NS && NR == Mech_JA919::NR)
        k_react_queue_batch<NS, Mech_JA919><<<grid, 128, 0, a.stream>>>(*a.mech, tab, n, next, a.max_substeps,
                                                                        counter);
    else
        k_react_queue_batch<NS, TableRates<NS, NR>><<<grid, 128, 0, a.stream>>>(*a.mech, tab, n, next,
                                                                                a.max_substeps, counter);
    return cudaGetLastError();
}

#ifdef EU_MIXED // the FP64 flavours' deferred cells stay in their instance's branch
template <int NS, int NR>
cudaError_t heavy_batch_t(const LaunchArgs &a, const BatchCell *tab, int n, int *next, int blocks)
{
    k_react_heavy_batch<NS, NR><<<dim3(unsigned(blocks)), 128, 0, a.stream>>>(*a.mech, tab, n, next + 1,
                                                                               a.max_substeps);
    return cudaGetLastError();
}
#endif

} // namespace

// Supported (NS, NR): the repository mechanism H2_JA919 (9 species, 19
// reactions), the one the reference's parser reads.
#define EU3D_DISPATCH(fn, ...)                                                                     \
    switch (a.mech->ns * 100 + a.mech->nr) {                                                        \
    case 919:                                                                                      \
        return fn<9, 19>(__VA_ARGS__);                                                             \
    default:                                                                                       \
        return cudaErrorInvalidValue;                                                              \
    }

cudaError_t launch_boundary(const LaunchArgs &a) { EU3D_DISPATCH(boundary_t, a) }
cudaError_t launch_flux_update(const LaunchArgs &a) { EU3D_DISPATCH(flux_t, a) }
int flux_plan(const LaunchArgs &a)
{
#ifdef EU_MIXED
    if (takes_tiled(a))
        return tiled_ci(a);
#endif
    return small_grid(a) ? -1 : 0;
}
cudaError_t launch_recover_react(const LaunchArgs &a, bool react) { EU3D_DISPATCH(react_t, a, react) }
cudaError_t launch_derived(const LaunchArgs &a, int which, double *out) { EU3D_DISPATCH(derived_t, a, which, out) }
cudaError_t launch_materialize(const LaunchArgs &a) { EU3D_DISPATCH(materialize_t, a) }
cudaError_t launch_to_f32(const double *src, float *dst, long long n, cudaStream_t s)
{
    if (n <= 0)
        return cudaSuccess;
    k_to_f32<<<dim3(unsigned(std::min<long long>((n + 255) / 256, 148LL * 16))), 256, 0, s>>>(src, dst, n);
    return cudaGetLastError();
}

cudaError_t launch_recover_classify(const LaunchArgs &a, const LearnedParams &lp) { EU3D_DISPATCH(classify_t, a, lp) }
cudaError_t launch_learned_apply(const LaunchArgs &a, const LearnedParams &lp) { EU3D_DISPATCH(apply_t, a, lp) }
cudaError_t launch_learned_route(const LaunchArgs &a, const LearnedParams &lp) { EU3D_DISPATCH(route_t, a, lp) }
cudaError_t launch_react_queue(const LaunchArgs &a, const int *queue, int *count, int counter)
{
    EU3D_DISPATCH(react_queue_t, a, queue, count, counter)
}
cudaError_t launch_state_from_tpy(const LaunchArgs &a, long long n, const double *T, const double *p, const double *Y,
                                  double *cs, double *E)
{
    EU3D_DISPATCH(state_from_tpy_t, a, n, T, p, Y, cs, E)
}
#ifdef EU_EXACT_RATES
cudaError_t launch_chem_samples(const LaunchArgs &a, long long n, double *cs, double *T, double *E, const double *dt,
                                int *nchem, int *heavy)
{
    EU3D_DISPATCH(chem_samples_t, a, n, cs, T, E, dt, nchem, heavy)
}
#endif

cudaError_t launch_react_heavy(const LaunchArgs &a, int blocks) { EU3D_DISPATCH(heavy_t, a, blocks) }
cudaError_t launch_react_queue_batch(const LaunchArgs &a, const BatchCell *tab, int n, int *next, int counter)
{
    EU3D_DISPATCH(react_queue_batch_t, a, tab, n, next, counter)
}
#ifdef EU_MIXED
cudaError_t launch_react_heavy_batch(const LaunchArgs &a, const BatchCell *tab, int n, int *next, int blocks)
{
    EU3D_DISPATCH(heavy_batch_t, a, tab, n, next, blocks)
}
constexpr auto react_heavy_batch = &launch_react_heavy_batch;
#else
constexpr decltype(Launchers::react_heavy_batch) react_heavy_batch = nullptr;
#endif

cudaError_t launch_cfl(const LaunchArgs &a, double cfl, unsigned long long *slot, double *time)
{
    const long long n = (long long)a.g.ni * a.g.nj * a.g.nk;
    const unsigned blocks = unsigned(std::min<long long>((n + 255) / 256, (long long)(a.sms > 0 ? a.sms : 148) * 8));
    k_cfl<<<blocks, 256, 0, a.stream>>>(a.g, a.st, slot, cfl, const_cast<double *>(a.dt_dev), time);
    return cudaGetLastError();
}

// face 0: x low, 1: x high; pack: planes -> msg, else msg -> ghost planes.
cudaError_t launch_halo(const LaunchArgs &a, int nf, int face, bool pack, void *msg)
{
    const DevGrid &g = a.g;
    const long long plane = (long long)g.ny * g.nz;
    int first, step;
    if (pack) {
        first = face == 0 ? g.bc + 1 : g.ni + g.bc - 2;
        step = face == 0 ? 1 : -1;
    } else {
        first = face == 0 ? g.bc - 1 : g.ni + g.bc;
        step = face == 0 ? -1 : 1;
    }
    const long long total = (long long)nf * g.bc * plane;
    const unsigned blocks = unsigned(std::min<long long>((total + 255) / 256, (long long)(a.sms > 0 ? a.sms : 148) * 8));
    if (a.st.prim32)
        k_halo_copy<float><<<blocks, 256, 0, a.stream>>>(a.st.prim32, static_cast<float *>(msg), nf, g.bc, g.n3, plane,
                                                       first, step, pack);
    else
        k_halo_copy<double><<<blocks, 256, 0, a.stream>>>(a.st.prim, static_cast<double *>(msg), nf, g.bc, g.n3, plane,
                                                        first, step, pack);
    return cudaGetLastError();
}

cudaError_t launch_rk_combine(const LaunchArgs &a, const double *cs0, double ca, double cb)
{
    const long long n = (long long)a.g.ni * a.g.nj * a.g.nk;
    const unsigned blocks = unsigned(std::min<long long>((n + 255) / 256, (long long)(a.sms > 0 ? a.sms : 148) * 8));
    k_rk_combine<<<blocks, 256, 0, a.stream>>>(a.g, a.st.cs, cs0, a.mech->ns + 4, ca, cb);
    return cudaGetLastError();
}

cudaError_t launch_set_value(double *dst, double v, cudaStream_t s)
{
    k_set_value<<<1, 1, 0, s>>>(dst, v);
    return cudaGetLastError();
}

const Launchers launchers = {&launch_boundary,         &launch_flux_update,      &launch_recover_react,
                             &launch_derived,          &launch_recover_classify, &launch_learned_apply,
                             &launch_react_queue,      &launch_react_heavy,      &launch_materialize,
                             &launch_learned_route,    &launch_react_queue_batch, react_heavy_batch,
                             &flux_plan};

#undef EU3D_DISPATCH

} // namespace EU3D_NS
} // namespace eu3d
