// eu3d_kernels.cuh — the timestep kernels, templated on the species and
// reaction counts. Instantiated three times: eu3d_kernels_strict.cu (--fmad=false,
// EU_EXACT_THERMO, EU_EXACT_RATES, EU_EXACT_FLUX), eu3d_kernels_fast.cu
// (EU_EXACT_THERMO) and eu3d_kernels_mixed.cu (EU_MIXED).
#pragma once

#include "eu3d_device.cuh"
#include "eu3d_mech_JA919.cuh"
#include "eu3d_tc.cuh"

#ifndef EU3D_NS
#error "define EU3D_NS (the arithmetic flavour's namespace) before including eu3d_kernels.cuh"
#endif

// Kernels live in a per-flavour namespace: the strict and fast translation
// units instantiate the same templates with different arithmetic, and their
// host-side symbols must not merge at link time.
namespace eu3d {
namespace EU3D_NS {

// ---------------------------------------------------------------- ghosts
// Flowfield::FieldBoundary_3dRSBI (src/Flowfield.cpp:593-807) on the ghost
// layers the stencils read: x faces over interior (j,k), y faces over interior
// (i,k), z faces over interior (i,j). One thread per ghost node.
//   x low/high: zero-gradient mirror copy      (:597-641)
//   y low: symmetry, V reflected, rho/H/Gamma rebuilt from mirrored T, p, Y (:647-679)
//   y high: zero-gradient mirror copy          (:684-705)
//   z low/high: mirror copy with W reflected   (:710-802)
// With g.bc_kind == 1 the x faces follow Flowfield::FieldBoundary_1dZND
// (src/Flowfield.cpp:317-411, commented out in the reference): x low a
// reflecting wall (mirror copy, U reflected), x high outflow (mirror copy of
// U, V, p, T, Y with rho/H/Gamma rebuilt as on the y-low face).
template <int NS>
__global__ void __launch_bounds__(256) k_boundary(const __grid_constant__ DevMech m, const DevGrid g,
                                                  const DevState st)
{
    if (blockIdx.x == 0 && threadIdx.x < kStepWords)
        st.step_words[threadIdx.x] = 0;
    const int bc = g.bc, ni = g.ni, nj = g.nj, nk = g.nk;
    // z ghosts of a row: on a grid two nodes thick every interior node is the
    // mirror source of one ghost below and one above, and a thread fills both
    // from one read and one rebuild (1024 x 512 x 2 ODW: 0.122 -> 0.093 ms)
    const bool both = nk == bc;
    const int zper = both ? bc : 2 * bc;
    const long long nxf = 2LL * bc * nj * nk, nyf = 2LL * bc * ni * nk, nzf = (long long)zper * ni * nj;
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nxf + nyf + nzf)
        return;
    const long long n3 = g.n3;
    long long dst, src;
    double su = 1, sv = 1, sw = 1;
    bool rebuild = false;
    long long inflow = -1; // ODW x-low: index into the inflow tables
    long long again = 0;   // distance to a second ghost of the same value
    if (t < nxf) {
        const int jk = fdiv(t, g.d_nk), q = fdiv(t, g.d_njnk); // q: 0 .. 2bc-1
        const int k = bc + int(t - (long long)jk * nk);
        const int j = bc + (jk - q * nj);
        if (q < bc ? g.exch_lo : g.exch_hi) // filled by the halo exchange
            return;
        const int i = q < bc ? q : ni + q;           // ghost index
        const int si = q < bc ? 2 * bc - 1 - i : 2 * (ni + bc) - 1 - i;
        dst = cell_index(g, i, j, k);
        src = cell_index(g, si, j, k);
        if (g.bc_kind == 1) {
            su = q < bc ? -1 : 1;
            rebuild = q >= bc;
        } else if (g.bc_kind == 2) { // ODW: freestream tables in, rebuilt outflow out
            if (q < bc)
                inflow = (long long)(j - bc) * nk + (k - bc);
            rebuild = q >= bc;
        }
    } else if (t < nxf + nyf) {
        t -= nxf;
        const int ik = fdiv(t, g.d_nk), q = fdiv(t, g.d_nink);
        const int k = bc + int(t - (long long)ik * nk);
        const int i = bc + (ik - q * ni);
        const int j = q < bc ? q : nj + q;
        const int sj = q < bc ? 2 * bc - 1 - j : 2 * (nj + bc) - 1 - j;
        dst = cell_index(g, i, j, k);
        src = cell_index(g, i, sj, k);
        if (q < bc) {
            if (g.bc_kind == 2 && i - bc < g.wall_i0) {
                inflow = k - bc; // ODW ahead of the wall: the freestream (first table row)
            } else {
                sv = -1;
                rebuild = true;
            }
        }
    } else {
        // the ghost index runs fastest: the 2 bc ghosts of one (i, j) row sit in
        // two contiguous pairs, so a warp touches 16 pairs instead of 32 rows
        t -= nxf + nyf;
        if (st.zm_fresh && *st.zm_fresh) // EU_GHOSTS_STORED: stored with the interior
            return;
        const int jq = fdiv(t, g.d_ghost), ii = fdiv(t, g.d_ghost_nj);
        const int q = int(t - (long long)jq * zper);
        again = both ? nk + bc : 0;
        const int j = bc + (jq - ii * nj);
        const int i = bc + ii;
        const int k = q < bc ? q : nk + q;
        const int sk = q < bc ? 2 * bc - 1 - k : 2 * (nk + bc) - 1 - k;
        dst = cell_index(g, i, j, k);
        src = cell_index(g, i, j, sk);
        sw = -1;
        rebuild = g.bc_kind == 2; // ODW rebuilds the thermo on the z faces
    }
    if (inflow >= 0) {
        const long long nt = (long long)nj * nk;
#pragma unroll
        for (int f = 0; f < 7 + NS; ++f) {
            const double v = st.inflow[f * nt + inflow];
            if (st.prim32)
                st.prim32[f * n3 + dst] = float(v);
            else
                st.prim[f * n3 + dst] = v;
        }
        st.T[dst] = st.inflow[(7 + NS) * nt + inflow];
        return;
    }
    // mixed precision keeps only the FP32 primitive planes current (the flux
    // kernel's input); the FP64 path its FP64 planes
    double v[7 + NS];
#pragma unroll
    for (int f = 0; f < 7 + NS; ++f) v[f] = st.prim32 ? double(st.prim32[f * n3 + src]) : st.prim[f * n3 + src];
    v[kU] = su * v[kU];
    v[kV] = sv * v[kV];
    v[kW] = sw * v[kW];
    const double T = st.T[src];
    if (rebuild) {
#ifndef EU_EXACT_THERMO
        double rg = 0, Y[NS];
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            Y[s] = v[kY0 + s];
            rg = fma(Y[s], m.ri[s], rg);
        }
        MixPoly<NS> mp;
        mix_poly<NS>(m, Y, T < kThermoSwitch, mp);
        const double Rgas = rg * 1000, inv = rcp_nr(T);
        const double h = fma(T, fma(T, fma(T, fma(T, fma(T, mp.h6, mp.h5), mp.h4), mp.h3), mp.a2), mp.a7) - mp.a0 * inv +
                         mp.a1 * log(T);
        const double cp = fma(T, fma(T, fma(T, fma(T, mp.a6, mp.a5), mp.a4), mp.a3), mp.a2) + inv * fma(mp.a0, inv, mp.a1);
        v[kD] = div_fast(v[kP], T * Rgas);
        v[kH] = h * 1000;
        v[kG] = div_fast(cp * 1000, cp * 1000 - Rgas);
#else
        const TPow p = make_tpow(T, true);
        double rg = 0, cp = 0, h = 0, e = 0;
        double Cpi[NS], Hi[NS];
        by_range(p.low, [&](auto range) {
            constexpr int kR = decltype(range)::value;
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                Cpi[s] = cp_species<NS, kR>(m, p, m.ri[s], s);
                Hi[s] = h_species<NS, kR>(m, p, m.ri[s], s);
            }
        });
#pragma unroll
        for (int s = 0; s < NS; ++s) rg += v[kY0 + s] * m.ri[s];
        const double Rgas = rg * 1000;
        v[kD] = v[kP] / (T * Rgas);
#pragma unroll
        for (int s = 0; s < NS; ++s) cp += Cpi[s] * v[kY0 + s];
#pragma unroll
        for (int s = 0; s < NS; ++s) h += v[kY0 + s] * Hi[s];
        (void)e;
        const double Cp = cp * 1000;
        v[kH] = h * 1000;
        v[kG] = Cp / (Cp - Rgas);
#endif
    }
    for (;;) {
        st.T[dst] = T;
#pragma unroll
        for (int f = 0; f < 7 + NS; ++f) {
            if (st.prim32)
                st.prim32[f * n3 + dst] = float(v[f]);
            else
                st.prim[f * n3 + dst] = v[f];
        }
        if (!again)
            break;
        dst += again;
        again = 0;
    }
}

// Halo messages between x blocks (Flowfield::Mpi_Boundary, src/Flowfield.cpp:809-911):
// plane p (0 .. bc-1) of field f of a message is node plane src_i(p) of the flux
// primitives. to_msg: planes -> message (pack), else message -> planes (unpack).
// Node planes: pack face 0 takes bc+1+p, pack face 1 takes ni+bc-2-p; unpack
// face 0 fills bc-1-p, unpack face 1 fills ni+bc+p.
template <typename R>
__global__ void k_halo_copy(R *planes, R *msg, int nf, int bc, long long n3, long long plane, int first, int step,
                            bool to_msg)
{
    const long long total = (long long)nf * bc * plane;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const long long fp = t / plane, e = t - fp * plane;
        const int f = int(fp / bc), p = int(fp - (long long)f * bc);
        R *node = planes + f * n3 + (long long)(first + step * p) * plane + e;
        if (to_msg)
            msg[t] = *node;
        else
            *node = msg[t];
    }
}

// ----------------------------------------------------------------- fluxes

// Tile of k_flux_update_faces: cells per axis, the divisions of its flat face
// lists, and the faces they hold. Blocks are kFaceThreadsWide threads on grids
// that fill the chip once at most (a face a thread, one round), half of that
// on larger ones.
constexpr int kFaceThreads = 128, kFaceThreadsWide = 256;
// Flux slots of a component: the faces of a tile at most. 464 doubles are the
// most with which four 128-thread blocks share an SM (at 496 three do: 1.30 ms
// against 0.85 on 256 x 128 x 128).
template <typename R>
constexpr int kFacePitch = sizeof(R) == 8 ? 464 : 496;
struct FaceTile {
    int ti, tj, tk;
    bool y_first; // blockIdx.x counts the tiles along y and blockIdx.y those along z (more than 65,535 along y)
    FastDiv d_tk, d_tk1, d_area, d_area_y, d_area_z;
};

template <int NS, typename R>
constexpr size_t face_smem_bytes()
{
    return sizeof(R) * (NS + 4) * kFacePitch<R>;
}

// Flux divergence and the Euler-explicit update (TimeAdv::EE, src/TimeAdv.cpp:42-56,
// then CS += RHS, src/Flowfield.cpp:1350-1354) with one thread per face: every
// FP64 grid, and FP32 fluxes on thin or small grids.
//
// A block owns a ti x tj x tk tile of cells (chosen from the grid at run time,
// FaceTile), marches ci nodes along x in steps of ti, and per step forms the
// tile's x, y and z faces as one flat list (a face a thread at a time, stencil
// points through the read-only cache), leaves the fluxes in shared memory and
// updates the cells from them. The x faces above the last plane are carried to
// the next step. The RHS keeps the reference's order -dt/dx (F+ - F-) - dt/dy
// (G+ - G-) - dt/dz (Q+ - Q-): in FP64, or for R = float the differences and
// their sum in FP32 onto the FP64 conserved value.
//
// What bounds it: in FP64 the instruction issue (about 2/5 of the instructions
// are FP64 ones). A thread that forms one face needs a third of the state of one
// that forms a cell's three, so 16 warps fit an SM without spills where the
// cell-a-thread forms ran 8 at 255 registers, and a tile's shape follows the
// grid, where fixed 32-lane rows left most lanes idle on thin grids and a few
// blocks marched 16 planes one after the other on small ones. Flux phase of a
// step on a B200, before and after:
//   256 x 128 x 128 FP64  1.60 -> 0.85 ms    129 x 65 x 65 FP64   0.367 -> 0.133 ms
//   281 x 141 x 2 strict  0.92 -> 0.093 ms   33 x 17 x 17 strict  0.396 -> 0.023 ms
//   4001 x 2 x 2 FP64    0.448 -> 0.014 ms   41 x 24 x 23 FP64    0.144 -> 0.015 ms
//   1024 x 512 x 2 FP32   0.40 -> 0.18 ms    48 x 32 x 32 FP32    0.073 -> 0.020 ms
template <int NS, typename R, bool kStrict>
__global__ void __launch_bounds__(kFaceThreadsWide, 2)
    k_flux_update_faces(const DevGrid g, const DevState st, const R *__restrict__ prim,
                        const double *__restrict__ dt_dev, const FaceTile t, int ci)
{
    constexpr int NV = NS + 4, kPitch = kFacePitch<R>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R *sF = reinterpret_cast<R *>(smem_raw); // [NV][kPitch]
    const int tid = threadIdx.x, nthreads = blockDim.x;
    const int area = t.tj * t.tk; // cells of a plane
    const int nfx = (t.ti + 1) * area, nfy = t.ti * (t.tj + 1) * t.tk, nf = nfx + nfy + t.ti * t.tj * (t.tk + 1);
    const int k0 = (t.y_first ? blockIdx.y : blockIdx.x) * t.tk, j0 = (t.y_first ? blockIdx.x : blockIdx.y) * t.tj;
    const int rows = min(t.tj, g.nj - j0), cols = min(t.tk, g.nk - k0);
    const int i_begin = blockIdx.z * ci, i_end = min(i_begin + ci, g.ni);
    const long long n3 = g.n3;
    const int sx = g.ny * g.nz, sy = g.nz;
    const double dt = *dt_dev;
    for (int i0 = i_begin; i0 < i_end; i0 += t.ti) {
        const int planes = min(t.ti, i_end - i0);
        for (int f = tid + (i0 == i_begin ? 0 : area); f < nf; f += nthreads) {
            int dir, a, j, k, stride;
            bool in;
            if (f < nfx) {
                dir = 0;
                stride = sx;
                a = fdiv(f, t.d_area);
                const int r = f - a * area;
                j = fdiv(r, t.d_tk);
                k = r - j * t.tk;
                in = a <= planes && j < rows && k < cols;
                --a;
            } else if (f < nfx + nfy) {
                dir = 1;
                stride = sy;
                const int e = f - nfx;
                a = fdiv(e, t.d_area_y);
                const int r = e - a * (area + t.tk);
                j = fdiv(r, t.d_tk);
                k = r - j * t.tk;
                in = a < planes && j <= rows && k < cols;
                --j;
            } else {
                dir = 2;
                stride = 1;
                const int e = f - nfx - nfy;
                a = fdiv(e, t.d_area_z);
                const int r = e - a * (area + t.tj);
                j = fdiv(r, t.d_tk1);
                k = r - j * (t.tk + 1);
                in = a < planes && j < rows && k <= cols;
                --k;
            }
            if (in) {
                const R *p = prim + cell_index(g, g.bc + i0 + a, g.bc + j0 + j, g.bc + k0 + k) - stride;
                face_ausm_dir<NS, R, kStrict>(dir, p, unsigned(n3), stride, [&](int q, R v) { sF[q * kPitch + f] = v; });
            }
        }
        __syncthreads();
        for (int e = tid; e < t.ti * area; e += nthreads) {
            const int a = fdiv(e, t.d_area), r = e - a * area, j = fdiv(r, t.d_tk), k = r - j * t.tk;
            if (a >= planes || j >= rows || k >= cols)
                continue;
            const int i = g.bc + i0 + a, jj = g.bc + j0 + j, kk = g.bc + k0 + k;
            const long long c = cell_index(g, i, jj, kk);
            const double cx = -dt / (g.x[i] - g.x[i - 1]), cy = dt / (g.y[jj] - g.y[jj - 1]),
                         cz = dt / (g.z[kk] - g.z[kk - 1]);
            const int fx = e, fy = nfx + e + a * t.tk, fz = nfx + nfy + e + a * t.tj + j;
            double old[NV];
#pragma unroll
            for (int q = 0; q < NV; ++q) old[q] = st.cs[q * n3 + c];
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                const R *F = sF + q * kPitch;
                const R xp = F[fx + area], xm = F[fx], yp = F[fy + t.tk], ym = F[fy], zp = F[fz + 1], zm = F[fz];
                if constexpr (sizeof(R) == 4) {
                    const float rhs = float(cx) * float(xp - xm) - float(cy) * float(yp - ym) - float(cz) * float(zp - zm);
                    st.cs[q * n3 + c] = old[q] + double(rhs);
                } else {
                    const double rhs = cx * (xp - xm) - cy * (yp - ym) - cz * (zp - zm);
                    st.cs[q * n3 + c] = old[q] + rhs;
                }
            }
        }
        if (i0 + t.ti < i_end) {
            __syncthreads();
            for (int e = tid; e < NV * area; e += nthreads) {
                const int q = fdiv(e, t.d_area), r = e - q * area;
                sF[q * kPitch + r] = sF[q * kPitch + t.ti * area + r];
            }
            __syncthreads();
        }
    }
}

// Plane-tiled flux divergence and update (FP32 fluxes): the same faces and RHS
// order as k_flux_update_faces, with every primitive read from HBM once per
// plane instead of once per stencil point, and the loads of the next plane
// overlapped with the current plane's arithmetic.
//
// A block owns a kTileJ x kTileK tile of (j, k) columns and marches along x with
// kTileJ + 1 warps. Warps 0 .. kTileJ-1 own a row of cells each: every thread
// keeps its column's x-stencil (planes i-1 .. i+2 of every primitive) in
// registers and loads plane i+3 one node ahead. Plane i of the tile plus a
// two-node halo in j and k is staged in shared memory, from which the y- and
// z-face fluxes are formed; two stages alternate, and while plane i is computed
// the halo of plane i+1 (cp.async) is in flight. The update of a plane waits for
// the next plane's barrier, so a plane has one (the face fluxes lie twice), and
// is an FP64 addition that the L2 carries out. sG: [r] the y face below
// tile row r (r = kTileJ: above the last row); sQ: [r][c] the z face left
// of column c.
//
// What bounds it is instruction issue (57 % active at 16 warps per SM). With two
// barriers a plane, the conserved values staged by cp.async and 64-bit node
// numbers it took 0.459 ms at 256 x 128 x 128 (278 M warp instructions); now
// 0.403 ms, the same bits. The addresses count most of that: a node number of 32 bits
// and a plane's offset as one wide multiply-add (0.460 -> 0.403 ms).
//
// Each cell warp forms three faces per plane (x, y, z). The edge warp (warp
// kTileJ) owns the first halo row above the tile, which it stages from its
// registers, and forms the two faces a full tile has beyond its cells: the y
// faces above the last row and the z faces right of the last column. No warp
// forms a fourth face, so no warp waits at the plane's barrier for another's
// extra face. Partial tiles: the faces of the valid rows/columns are formed,
// including the one past the last valid row/column.
//
// Tile height: 7 cell rows (8 warps), so that two blocks fit per SM (99 KB of
// shared memory each).
constexpr int kTileK = 32, kTileCols = kTileK + 4;
constexpr int kTileJ = 7, kTileWarps = kTileJ + 1, kTileRows = kTileJ + 4;
// staged by cp.async: rows 0, 1 and kTileJ + 3 over the full width, and the two
// columns each side of rows 2 .. kTileJ + 2 (the cell rows and the edge warp's row)
constexpr int kTileHalo = 3 * kTileCols + 4 * (kTileJ + 1);

template <int NS>
constexpr size_t tiled_flux_smem_bytes()
{
    return sizeof(float) * 2 * ((7 + NS) * kTileRows * kTileCols +
                                (NS + 4) * ((kTileJ + 1) * kTileK + kTileJ * (kTileK + 1)));
}

// Face flux from four consecutive stencil points of the staged plane tile,
// starting at (r, c) and stepping (DR, DC). own: the values of stencil point 2
// when that point is the thread's own node (kept in registers), else null.
template <int NS, int DIR, int DR, int DC, bool kOwn>
__device__ __forceinline__ void tile_face_flux(const float (*sP)[kTileRows][kTileCols], int r, int c, const float *own,
                                               float (&F)[NS + 4])
{
    constexpr int S = DR * kTileCols + DC, N = kTileRows * kTileCols;
    const float *p = &sP[0][r][c];
    face_ausm<NS, DIR, float>([&](int f, int q) { return (kOwn && q == 2) ? own[f] : p[f * N + q * S]; },
                              [&](int f, bool up, float &u, float &w, float &v) {
                                  w = p[f * N + (up ? 0 : 3 * S)];
                                  if (kOwn) {
                                      const float a = p[f * N + S];
                                      u = up ? a : own[f];
                                      v = up ? own[f] : a;
                                  } else {
                                      u = p[f * N + (up ? S : 2 * S)];
                                      v = p[f * N + (up ? 2 * S : S)];
                                  }
                              },
                              F);
}

template <int NS>
__device__ __forceinline__ void window_face_flux(const float (&w)[4][7 + NS], float (&F)[NS + 4])
{
    face_ausm<NS, 0, float>([&](int f, int p) { return w[p][f]; },
                            [&](int f, bool up, float &u, float &o, float &v) {
                                u = up ? w[1][f] : w[2][f];
                                o = up ? w[0][f] : w[3][f];
                                v = up ? w[2][f] : w[1][f];
                            },
                            F);
}

template <int NS>
__global__ void __launch_bounds__(kTileK *kTileWarps, 2)
    k_flux_update_tiled(const DevGrid g, const DevState st, const float *__restrict__ prim,
                        const double *__restrict__ dt_dev, int ci)
{
    using R = float;
    constexpr int NP = 7 + NS, NV = NS + 4;
    using Plane = R[NP][kTileRows][kTileCols];
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using FacesY = R[NV][kTileJ + 1][kTileK];
    using FacesZ = R[NV][kTileJ][kTileK + 1];
    Plane *stage = reinterpret_cast<Plane *>(smem_raw);
    FacesY *sG2 = reinterpret_cast<FacesY *>(stage + 2);
    FacesZ *sQ2 = reinterpret_cast<FacesZ *>(sG2 + 2);
    __shared__ float sX[2]; // -dt / dx of a plane

    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * kTileK + tx;
    const int k0 = blockIdx.x * kTileK, j0 = blockIdx.y * kTileJ;
    const int k = g.bc + k0 + tx, j = g.bc + j0 + ty;
    const int rows = min(kTileJ, g.nj - j0), cols = min(kTileK, g.nk - k0); // valid rows / columns
    const bool valid = ty < rows && tx < cols;
    const bool resident = j < g.ny && k < g.nz; // inside the haloed arrays: staged for the neighbours
    // faces this thread forms (see above); the y face above a full tile's
    // last row is the edge warp's (ty == rows == kTileJ)
    const bool yface = tx < cols && ty <= rows;
    const bool zface = ty < rows && tx <= cols;
    const int zrow = tx; // lanes 0..kTileJ-1 of the edge warp: the z face right of the last column
    const bool zright = ty == kTileJ && zrow < rows && cols == kTileK;

    // the halo cell this thread stages, if any (counted from the last thread,
    // so the edge warp, which forms fewer faces, takes the first share)
    int hr = -1, hc = 0;
    {
        const int h = kTileWarps * kTileK - 1 - tid;
        if (h < 3 * kTileCols) {
            const int band = h / kTileCols;
            hr = band < 2 ? band : kTileJ + 3;
            hc = h % kTileCols;
        } else if (h < kTileHalo) {
            const int e = h - 3 * kTileCols, side = e % 4;
            hr = 2 + e / 4;
            hc = side < 2 ? side : kTileK + side;
        }
    }
    const int hj = g.bc + j0 - 2 + hr, hk = g.bc + k0 - 2 + hc;
    const bool halo = hr >= 0 && hj < g.ny && hk < g.nz;

    // node numbers fit 32 bits; a plane times n3 is formed in 64
    const unsigned n3 = unsigned(g.n3), sx = unsigned(g.ny) * unsigned(g.nz);
    auto node = [&](const R *base, int f, unsigned c) {
        return reinterpret_cast<const R *>(reinterpret_cast<const char *>(base + c) +
                                           (unsigned long long)n3 * unsigned(f * int(sizeof(R))));
    };
    const double dt = *dt_dev;
    const float cy32 = valid ? float(dt / (g.y[j] - g.y[j - 1])) : 0.0f;
    const float cz32 = valid ? float(dt / (g.z[k] - g.z[k - 1])) : 0.0f;
    const int i_begin = g.bc + blockIdx.z * ci;
    const int i_end = min(i_begin + ci, g.bc + g.ni);
    const unsigned col = resident ? unsigned(cell_index(g, 0, j, k)) : 0;
    const unsigned hcol = halo ? unsigned(cell_index(g, 0, hj, hk)) : 0;

    // plane p of the tile into stage s: the own node from registers, the halo
    // node by cp.async; one commit group per call (empty when nothing to copy)
    auto stage_plane = [&](int p, const R(&own)[NP], int s) {
        if (resident) {
#pragma unroll
            for (int f = 0; f < NP; ++f) stage[s][f][ty + 2][tx + 2] = own[f];
        }
        if (halo) {
#pragma unroll
            for (int f = 0; f < NP; ++f) tc::cp_async4(&stage[s][f][hr][hc], node(prim, f, hcol + unsigned(p) * sx));
        }
        tc::cp_async_commit();
    };

    R w[4][NP];
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int f = 0; f < NP; ++f) w[p][f] = resident ? __ldg(node(prim, f, col + unsigned(i_begin - 2 + p) * sx)) : R(0);
    R Fm[NV];
    if (valid)
        window_face_flux<NS>(w, Fm);
#pragma unroll
    for (int f = 0; f < NP; ++f) {
        w[0][f] = w[1][f];
        w[1][f] = w[2][f];
        w[2][f] = w[3][f];
        w[3][f] = resident ? __ldg(node(prim, f, col + unsigned(i_begin + 2) * sx)) : R(0);
    }
    stage_plane(i_begin, w[1], 0);
    R dF[NV]; // F_{i+1/2} - F_{i-1/2} of the plane whose update is due

    for (int i = i_begin;; ++i) {
        // window: planes i-1, i, i+1, i+2. One barrier a plane: it shows plane i's
        // halo (stage s) and the y and z faces of plane i-1 (the other pair of
        // face arrays), and closes the reads of plane i-1's stage and of plane
        // i-2's faces, which this iteration overwrites.
        const int s = (i - i_begin) & 1;
        tc::cp_async_wait<0>();
        __syncthreads();
        if (i > i_begin && valid) { // update plane i-1
            const auto &sG = sG2[s ^ 1];
            const auto &sQ = sQ2[s ^ 1];
            const unsigned c = col + unsigned(i - 1) * sx;
            const float cx32 = sX[s ^ 1];
            // the flux differences and their sum in FP32 (a difference of two
            // FP32 values within a factor of two is exact), accumulated onto
            // the FP64 conserved value by the L2: nothing waits for its read
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                const float rhs = cx32 * dF[q] - cy32 * float(sG[q][ty + 1][tx] - sG[q][ty][tx]) -
                                  cz32 * float(sQ[q][ty][tx + 1] - sQ[q][ty][tx]);
                atomicAdd(reinterpret_cast<double *>(reinterpret_cast<char *>(st.cs + c) +
                                                     (unsigned long long)n3 * unsigned(q * int(sizeof(double)))),
                          double(rhs));
            }
        }
        if (i == i_end)
            break;
        auto &sG = sG2[s];
        auto &sQ = sQ2[s];
        if (i + 1 < i_end)
            stage_plane(i + 1, w[2], s ^ 1);
        if (yface) {
            R G[NV];
            tile_face_flux<NS, 1, 1, 0, true>(stage[s], ty, tx + 2, w[1], G);
#pragma unroll
            for (int q = 0; q < NV; ++q) sG[q][ty][tx] = G[q];
        }
        if (zface) {
            R Q[NV];
            tile_face_flux<NS, 2, 0, 1, true>(stage[s], ty + 2, tx, w[1], Q);
#pragma unroll
            for (int q = 0; q < NV; ++q) sQ[q][ty][tx] = Q[q];
        }
        if (zright) {
            R Q[NV];
            tile_face_flux<NS, 2, 0, 1, false>(stage[s], zrow + 2, kTileK, nullptr, Q);
#pragma unroll
            for (int q = 0; q < NV; ++q) sQ[q][zrow][kTileK] = Q[q];
        }
        R next[NP];
        const bool more = resident && i + 1 < i_end;
#pragma unroll
        for (int f = 0; f < NP; ++f) next[f] = more ? __ldg(node(prim, f, col + unsigned(i + 3) * sx)) : R(0);
        if (valid) {
            R Fp[NV];
            window_face_flux<NS>(w, Fp);
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                dF[q] = Fp[q] - Fm[q];
                Fm[q] = Fp[q];
            }
        }
        if (tid == kTileWarps * kTileK - 1)
            sX[s] = float(-dt / (g.x[i] - g.x[i - 1]));
#pragma unroll
        for (int f = 0; f < NP; ++f) {
            w[0][f] = w[1][f];
            w[1][f] = w[2][f];
            w[2][f] = w[3][f];
            w[3][f] = next[f];
        }
    }
}

// ------------------------------------------------- recovery + kinetics

// kWriteCs false: the conserved planes are unchanged (recovery alone reads
// them and changes nothing there), so they are not written back.
// tcache: the recovery's thermo sums for this state, or null.
template <int NS, bool kWriteCs = true>
__device__ __forceinline__ void store_cell(const DevMech &m, const DevState &st, long long n3, long long c,
                                           const CellState<NS> &cell, const ThermoCache<NS> *tcache = nullptr)
{
    double P, H, G;
    finish_primitives<NS>(m, cell, tcache, P, H, G);
    const double v[7] = {P, cell.D, cell.U, cell.V, cell.W, H, G};
    if (st.prim32) { // mixed precision: the FP64 planes are formed on demand (k_materialize)
#pragma unroll
        for (int f = 0; f < 7; ++f) st.prim32[f * n3 + c] = float(v[f]);
#pragma unroll
        for (int s = 0; s < NS; ++s) st.prim32[(kY0 + s) * n3 + c] = float(cell.Y[s]);
    } else {
#pragma unroll
        for (int f = 0; f < 7; ++f) st.prim[f * n3 + c] = v[f];
#pragma unroll
        for (int s = 0; s < NS; ++s) st.prim[(kY0 + s) * n3 + c] = cell.Y[s];
    }
    if (kWriteCs) {
#pragma unroll
        for (int q = 0; q < NS + 4; ++q) st.cs[q * n3 + c] = cell.cs[q];
    }
    st.T[c] = cell.T;
    st.E[c] = cell.E;
    if (!(isfinite(cell.D) && isfinite(cell.T)))
        atomicAdd(&st.counters[kCntNonfinite], 1ULL);
    if (st.zm_fresh) {
        // EU_GHOSTS_STORED: the z-face ghosts this node is the mirror source
        // of (k_boundary's z faces: ghost 2 bc - 1 - k below, 2 (nk + bc) - 1 -
        // k above, W reflected), the values the ghost fill would copy, in the
        // same 32-byte sectors as the node's own stores
        const long long row = fdiv(c, st.zm_dnz);
        const int k = int(c - row * st.zm_nz), bc = st.zm_bc, nk = st.zm_nk;
        auto mirror = [&](long long gc) {
            if (st.prim32) {
#pragma unroll
                for (int f = 0; f < 7; ++f) st.prim32[f * n3 + gc] = float(f == kW ? -v[f] : v[f]);
#pragma unroll
                for (int s = 0; s < NS; ++s) st.prim32[(kY0 + s) * n3 + gc] = float(cell.Y[s]);
            } else {
#pragma unroll
                for (int f = 0; f < 7; ++f) st.prim[f * n3 + gc] = f == kW ? -v[f] : v[f];
#pragma unroll
                for (int s = 0; s < NS; ++s) st.prim[(kY0 + s) * n3 + gc] = cell.Y[s];
            }
            st.T[gc] = cell.T;
        };
        if (k < 2 * bc)
            mirror(c + (2 * bc - 1 - 2 * k));
        if (k >= nk)
            mirror(c + (2 * (nk + bc) - 1 - 2 * k));
    }
}

// EU_GHOSTS_STORED: a recovery that stores every interior node has written
// every z-face ghost, so the next ghost fill (after it in stream order) may
// skip the z faces.
__device__ __forceinline__ void mark_z_fresh(const DevState &st)
{
    if (st.zm_fresh && blockIdx.x == 0 && threadIdx.x == 0)
        *st.zm_fresh = 1;
}

// Post-advection state recovery (Flowfield::Update_after_Adv ->
// Update_after_CS, src/Flowfield.cpp:1579-1617), Nchem prediction
// (Reaction::TrapezoidPrediction, src/Reaction.cpp:865-942) and the Nchem
// trapezoid substeps with state recovery after each (src/Euler.cpp:462-493,
// src/Reaction.cpp:562-805, src/Flowfield.cpp:1521-1536). The prediction's
// rate evaluation is reused by the first substep: both evaluate the same
// expression on the same state. One thread per interior node.
// Rate evaluation from the runtime tables (any mechanism of these sizes).
template <int NS_, int NR_>
struct TableRates {
    static constexpr int NS = NS_, NR = NR_;
    __device__ __forceinline__ static void rates(const DevMech &m, double T, double inv, double lnT,
                                                 const double (&mc)[NS], SpeciesRates<NS> &k)
    {
        eval_rates<NS, NR>(m, T, inv, lnT, mc, k);
    }
};

// Nchem prediction (Reaction::TrapezoidPrediction, src/Reaction.cpp:865-942)
// and the Nchem trapezoid substeps with state recovery after each
// (src/Euler.cpp:462-493, src/Reaction.cpp:562-805, src/Flowfield.cpp:1521-1536)
// on a recovered cell state. The prediction's rate evaluation is reused by
// the first substep: both evaluate the same expression on the same state.
// Returns Nchem; a prediction <= 0 or above max_substeps is counted as an error.
// Nchem = ceil(dtm / min_s |Di_s / Wi_s|) over species with Y_s >= 1e-6
// (src/Reaction.cpp:919-940); a prediction <= 0 or above max_substeps is bad
// (counted as an error) and gives 0 or max_substeps.
__device__ __forceinline__ int nchem_from_dt(double dtm, double dt, int max_substeps, bool &bad)
{
    const double ratio = ceil(dtm / dt);
    bad = !(ratio >= 1.0) || ratio > double(max_substeps);
    if (bad)
        return (ratio > double(max_substeps)) ? max_substeps : 0;
    return int(ratio);
}

// The threads that arrive here together with the same pointer (in a batch's
// shared stage a warp's cells may belong to several instances).
__device__ __forceinline__ unsigned peers(const void *p)
{
    const unsigned here = __activemask();
    int same;
    __match_all_sync(here, reinterpret_cast<unsigned long long>(p), &same);
    return same ? here : __match_any_sync(here, reinterpret_cast<unsigned long long>(p));
}

// The statistics of the cells' predictions, by the kernel that advances them:
// one set of atomics for the threads that arrive together. (One a cell on the
// two counters, all on one L2 slice, were what the kinetics waited for: 545,025
// cells of one substep each took 0.75 ms with the rates in either form, 0.26
// with a set a warp.)
__device__ __forceinline__ void count_nchem(unsigned long long *counters, int nchem, bool bad)
{
    const unsigned here = peers(counters);
    const unsigned errors = __ballot_sync(here, bad);
    const int most = __reduce_max_sync(here, nchem);
    const unsigned sum = __reduce_add_sync(here, unsigned(nchem)); // 32 x 2^20 at most by default
    const bool big = most >= (1 << 26);
    if (big) { // max_substeps beyond the sum's range: a cell at a time
        if (nchem > 0)
            atomicAdd(&counters[kCntSumNchem], (unsigned long long)nchem);
    }
    if ((threadIdx.x & 31) == __ffs(here) - 1) {
        if (errors)
            atomicAdd(&counters[kCntBadNchem], (unsigned long long)__popc(errors));
        if (most > 0) {
            if (!big)
                atomicAdd(&counters[kCntSumNchem], (unsigned long long)sum);
            if (*(volatile unsigned long long *)&counters[kCntMaxNchem] < (unsigned long long)most)
                atomicMax(&counters[kCntMaxNchem], (unsigned long long)most);
        }
    }
}

// One more on a counter for every thread that arrives.
__device__ __forceinline__ void count_threads(unsigned long long *counter)
{
    const unsigned here = peers(counter);
    if ((threadIdx.x & 31) == __ffs(here) - 1)
        atomicAdd(counter, (unsigned long long)__popc(here));
}

// The prediction: start-of-step rates (kept in `rates` for the first substep)
// and Nchem.
template <int NS, class Rt>
__device__ __forceinline__ int predict_nchem(const DevMech &m, const CellState<NS> &cell, double dtm,
                                             int max_substeps, bool &bad, double (&mc)[NS],
                                             SpeciesRates<NS> &rates)
{
    scaled_concentrations<NS>(m, cell, mc);
    Rt::rates(m, cell.T, cell.inv, cell.lnT, mc, rates);
    double dt = dtm;
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        // formed for every species, then chosen: a select instead of a branch
        // that the cells diverge on
        const double w = rates.w(m, s);
#ifdef EU_EXACT_RATES
        const double dt_temp = fabs(-(cell.cs[s] * 1e-3) / w);
#else
        const double dt_temp = fabs(cell.cs[s] * 1e-3 * rcp_nr(w));
#endif
        dt = (cell.Y[s] >= 1e-6 && w != 0 && dt_temp < dt) ? dt_temp : dt;
    }
    return nchem_from_dt(dtm, dt, max_substeps, bad);
}

// The Nchem substeps, the first one on the prediction's rates.
template <int NS, class Rt>
__device__ __forceinline__ void run_substeps(const DevMech &m, CellState<NS> &cell, double dtm, int nchem,
                                             double (&mc)[NS], SpeciesRates<NS> &rates, double *cms,
                                             long long cms_stride, ThermoCache<NS> &tcache)
{
    const double dts = dtm / nchem;
    for (int step = 0; step < nchem; ++step) {
        if (step > 0) {
            scaled_concentrations<NS>(m, cell, mc);
            Rt::rates(m, cell.T, cell.inv, cell.lnT, mc, rates);
        }
        if (cms) {
#pragma unroll
            for (int s = 0; s < NS; ++s) cms[s * cms_stride] = rates.w(m, s) * 1e3;
        }
        trapezoid_substep<NS>(m, rates, dts, mc, cell, tcache);
    }
}

// Cells whose predicted Nchem exceeds kHeavyNchem are deferred to k_react_heavy:
// one warp per cell instead of one thread, so the long serial substep chains of
// igniting cells do not set the step's time. st.heavy = {count, next, cells...}
// (null: every cell on its own thread). On the 48x32x32 igniting block in mixed
// precision the step took 0.865 / 0.81 / 0.764 / 0.78 / 1.11 ms with the
// threshold at 16 / 8 / 4 / 2 / 0: below 4 a warp per cell costs more than the
// few substeps it shortens. The other forms, at 16 / 8 / 4: strict igniting blocks of
// 41x24x23 and 96x48x48, 0.396 / 0.314 / 0.262 and 0.698 / 0.613 / 0.566 ms a step;
// fast FP64, ten steps of the smaller one with its copies, 4.75 / 4.19 / 3.99 ms;
// 100,000 chemistry samples, whose longest chain decides, 21.9 / 20.7 / 21.3 ms.
constexpr int kHeavyNchem = 4;

__device__ __forceinline__ void push_heavy(int *heavy, long long c)
{
    const unsigned here = peers(heavy), lane = threadIdx.x & 31;
    const int first = __ffs(here) - 1;
    int q = 0;
    if (int(lane) == first)
        q = atomicAdd(&heavy[0], __popc(here));
    q = __shfl_sync(here, q, first) + __popc(here & ((1u << lane) - 1));
    heavy[2 + q] = int(c);
}

// React one recovered cell, or (heavy queue present) defer it when its Nchem is
// large. Returns false when deferred. tcache: the last substep's thermo sums out.
template <int NS, class Rt>
__device__ __forceinline__ bool react_or_defer(const DevMech &m, const DevState &st, long long n3, long long c,
                                               CellState<NS> &cell, double dtm, int max_substeps,
                                              ThermoCache<NS> &tcache)
{
    double mc[NS];
    SpeciesRates<NS> rates;
    bool bad;
    load_temperature<NS>(cell, cell.T); // as a cell loaded from a queue
    const int nchem = predict_nchem<NS, Rt>(m, cell, dtm, max_substeps, bad, mc, rates);
    if (st.heavy && nchem > kHeavyNchem) {
        push_heavy(st.heavy, c);
        return false;
    }
    count_nchem(st.counters, nchem, bad);
    run_substeps<NS, Rt>(m, cell, dtm, nchem, mc, rates, st.cms ? st.cms + c : nullptr, n3, tcache);
    st.nchem[c] = nchem;
    return true;
}

template <int NS>
__device__ __forceinline__ void load_cell(const DevState &st, long long n3, long long c, CellState<NS> &cell)
{
#pragma unroll
    for (int q = 0; q < NS + 4; ++q) cell.cs[q] = st.cs[q * n3 + c];
    load_temperature<NS>(cell, st.T[c]);
    cell.E = st.E[c];
}

// The recovered state of a cell whose recovery already ran and was stored:
// D, Y, u, v, w are re-formed from CS with the expressions of recover_state
// (same values), T and E are the stored ones.
template <int NS>
__device__ __forceinline__ void load_recovered(const DevState &st, long long n3, long long c, CellState<NS> &cell)
{
    load_cell<NS>(st, n3, c, cell);
    double D = 0;
#pragma unroll
    for (int s = 0; s < NS; ++s) D += cell.cs[s];
    cell.D = D;
#ifdef EU_EXACT_THERMO
#pragma unroll
    for (int s = 0; s < NS; ++s) cell.Y[s] = cell.cs[s] / D;
    cell.U = cell.cs[NS + 0] / D;
    cell.V = cell.cs[NS + 1] / D;
    cell.W = cell.cs[NS + 2] / D;
#else
    const double invD = rcp_nr(D);
#pragma unroll
    for (int s = 0; s < NS; ++s) cell.Y[s] = cell.cs[s] * invD;
    cell.U = cell.cs[NS + 0] * invD;
    cell.V = cell.cs[NS + 1] * invD;
    cell.W = cell.cs[NS + 2] * invD;
#endif
}

// Mixed precision keeps the FP64 primitive planes out of the timestep (the
// FP32 planes feed the fluxes). This forms them on demand, for output: interior
// nodes from the stored conserved state, T and E (the values the FP64 store
// would have written), ghost nodes from the FP32 ghost planes.
template <int NS>
__global__ void __launch_bounds__(128) k_materialize(const __grid_constant__ DevMech m, const DevGrid g,
                                                     const DevState st)
{
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.n3)
        return;
    const long long n3 = g.n3;
    const int jk = fdiv(c, g.d_nz), i = fdiv(c, g.d_nynz);
    const int k = int(c - (long long)jk * g.nz), j = jk - i * g.ny;
    const bool interior = i >= g.bc && i < g.bc + g.ni && j >= g.bc && j < g.bc + g.nj && k >= g.bc &&
                          k < g.bc + g.nk;
    if (!interior) {
#pragma unroll
        for (int f = 0; f < 7 + NS; ++f) st.prim[f * n3 + c] = double(st.prim32[f * n3 + c]);
        return;
    }
    CellState<NS> cell;
    load_recovered<NS>(st, n3, c, cell);
    double P, H, G;
    finish_primitives<NS>(m, cell, P, H, G);
    const double v[7] = {P, cell.D, cell.U, cell.V, cell.W, H, G};
#pragma unroll
    for (int f = 0; f < 7; ++f) st.prim[f * n3 + c] = v[f];
#pragma unroll
    for (int s = 0; s < NS; ++s) st.prim[(kY0 + s) * n3 + c] = cell.Y[s];
}

// FP32 copy of the FP64 primitive planes (state upload in mixed precision).
__global__ void k_to_f32(const double *__restrict__ src, float *__restrict__ dst, long long n)
{
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        dst[t] = float(src[t]);
}

// Post-advection state recovery (Flowfield::Update_after_Adv ->
// Update_after_CS, src/Flowfield.cpp:1579-1617) followed, in the stiff modes,
// by the kinetics (react_or_defer). One thread per interior node.
// MINB: resident 128-thread blocks per SM the register allocation aims at
// (2: no spills, 8 warps; 3 and 4 trade spills for warps; the autotuner picks).
template <int NS, int NR, bool kReact, class Rt, int MINB = 2>
__global__ void __launch_bounds__(128, MINB) k_recover_react(const __grid_constant__ DevMech m, const DevGrid g,
                                                       const DevState st, const double *__restrict__ dt_dev,
                                                       int max_substeps)
{
    const long long ncell = (long long)g.ni * g.nj * g.nk;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    mark_z_fresh(st);
    if (t >= ncell)
        return;
    int i, j, k;
    interior_node(g, t, i, j, k);
    const long long n3 = g.n3;
    const long long c = cell_index(g, i, j, k);
    CellState<NS> cell;
    load_cell<NS>(st, n3, c, cell);
    ThermoCache<NS> recovered;
    recover_state<NS>(m, cell, recovered);
    if (!kReact) {
        store_cell<NS, false>(m, st, n3, c, cell, &recovered);
        return;
    }
    ThermoCache<NS> tcache;
    if (react_or_defer<NS, Rt>(m, st, n3, c, cell, *dt_dev, max_substeps, tcache))
        store_cell<NS>(m, st, n3, c, cell, &tcache);
    else
        store_cell<NS, false>(m, st, n3, c, cell); // recovered state for k_react_heavy
}

// ------------------------------------------------- learned chemistry

// Post-advection recovery of every cell; cells with chemistry to do are
// appended to the learned queue (warp-aggregated atomics), the others are
// final. Every cell's recovered state is stored.
// MINB: resident blocks per SM the register allocation aims at (the
// autotuner picks the instantiation; fewer registers, more warps, some spills).
template <int NS, int MINB = 4>
__global__ void __launch_bounds__(128, MINB) k_recover_classify(const __grid_constant__ DevMech m, const DevGrid g,
                                                          const DevState st, LearnedParams lp)
{
    const long long ncell = (long long)g.ni * g.nj * g.nk;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    mark_z_fresh(st);
    bool active = false;
    long long c = 0;
    if (t < ncell) {
        int i, j, k;
        interior_node(g, t, i, j, k);
        const long long n3 = g.n3;
        c = cell_index(g, i, j, k);
        CellState<NS> cell;
        load_cell<NS>(st, n3, c, cell);
        ThermoCache<NS> tcache;
        recover_state<NS>(m, cell, tcache);
        store_cell<NS, false>(m, st, n3, c, cell, &tcache);
        double reactive = 0, radical = 0;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            if (!lp.inert[s])
                reactive += cell.Y[s];
            if (lp.radical[s])
                radical += cell.Y[s];
        }
        active = reactive >= lp.frozen_y && !(cell.T < lp.frozen_T && radical < lp.frozen_radical);
        st.nchem[c] = 0;
    }
    const unsigned mask = __ballot_sync(0xffffffffu, active);
    if (mask) {
        const int lane = threadIdx.x & 31;
        int base = 0;
        if (lane == __ffs(mask) - 1)
            base = atomicAdd(&lp.counts[0], __popc(mask));
        base = __shfl_sync(0xffffffffu, base, __ffs(mask) - 1);
        if (active)
            lp.queue[base + __popc(mask & ((1u << lane) - 1))] = int(c);
    }
}

// Model inputs of the cell at position q of the model's queue: T, log10 p, Y_0 ..
// Y_{NS-1}, log10 dt, with p = rho R T and R = 8314.34 / Wav (Update_after_CS,
// src/Flowfield.cpp:1606-1608).
template <int NS>
__device__ __forceinline__ void learned_features(const DevMech &m, const LearnedParams &lp, long long q,
                                                 const CellState<NS> &cell, double dt)
{
    float *f = lp.feat + q * (NS + 3);
    double inv_w = 0;
#pragma unroll
    for (int s = 0; s < NS; ++s) inv_w += cell.Y[s] / m.mw[s];
    f[0] = float(cell.T);
    f[1] = float(log10(cell.T * cell.D * (kRUniv * 1000 * inv_w)));
#pragma unroll
    for (int s = 0; s < NS; ++s) f[2 + s] = float(cell.Y[s]);
    f[NS + 2] = float(log10(dt));
}

// Apply the ensemble's prediction to each queued cell, or send it to the stiff
// fallback queue. Accepted when every input lies in the trained box and the
// members' spread (largest per-output standard deviation, in output-scale
// units) is below tau. The mean species change is projected onto element
// conservation (which implies sum Y = 1), clipped at zero and renormalised;
// density, momentum and internal energy are held (the reference's chemistry
// changes only the species densities); T is re-solved by the Newton inversion
// from the predicted T.
template <int NS>
__global__ void __launch_bounds__(128) k_learned_apply(const __grid_constant__ DevMech m, const DevGrid g,
                                                       const DevState st, LearnedParams lp)
{
    // a fixed grid walks the queue in whole warps (the fallback append is
    // warp-aggregated)
    const int nq = lp.counts[0];
    const int stride = gridDim.x * blockDim.x;
    const int span = (nq + 31) / 32 * 32;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < span; q += stride) {
        bool fallback = false;
        int c = 0;
        if (q < nq) {
            const long long n3 = g.n3;
            c = lp.queue[q];
            const float *f = lp.feat + (long long)q * (NS + 3);
            bool ok = true;
#pragma unroll
            for (int a = 0; a < NS + 3; ++a) ok = ok && f[a] >= float(lp.box_lo[a]) && f[a] <= float(lp.box_hi[a]);
            double mean[NS + 1], spread = 0;
#pragma unroll
            for (int o = 0; o < NS + 1; ++o) {
                double s1 = 0, s2 = 0;
                for (int e = 0; e < lp.members; ++e) {
                    const double v = lp.pred[(long long)q * lp.pred_row + (long long)e * lp.pred_mem + o];
                    s1 += v;
                    s2 += v * v;
                }
                const double mu = s1 / lp.members;
                const double var = fmax(s2 / lp.members - mu * mu, 0.0);
                // spread and mean in the model's output space, the change back in physical units
                spread = fmax(spread, sqrt(var) * lp.out_scale[o]);
                mean[o] = lp.out_eps[o] > 0 ? lp.out_eps[o] * sinh(mu) : mu;
                ok = ok && (lp.out_bound[o] <= 0 || fabs(mean[o]) <= lp.out_bound[o]);
            }
            ok = ok && spread <= lp.tau && isfinite(spread);
            if (ok) {
                CellState<NS> cell;
                load_recovered<NS>(st, n3, c, cell);
                double dY[NS], Y[NS], sum = 0;
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    double d = 0;
#pragma unroll
                    for (int r = 0; r < NS; ++r) d += lp.proj[s][r] * mean[r];
                    dY[s] = d;
                }
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    Y[s] = fmax(cell.Y[s] + dY[s], 0.0);
                    sum += Y[s];
                }
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    cell.Y[s] = Y[s] / sum;
                    cell.cs[s] = cell.D * cell.Y[s];
                }
                load_temperature<NS>(cell, newton_temperature<NS>(m, cell.T + mean[NS], cell.E, cell.Y));
                store_cell<NS>(m, st, n3, c, cell);
                count_threads(&st.counters[kCntLearned]);
            } else {
                fallback = true;
            }
        }
        const unsigned mask = __ballot_sync(0xffffffffu, fallback);
        if (mask) {
            const int lane = threadIdx.x & 31;
            int base = 0;
            if (lane == __ffs(mask) - 1)
                base = atomicAdd(&lp.counts[1], __popc(mask));
            base = __shfl_sync(0xffffffffu, base, __ffs(mask) - 1);
            if (fallback)
                lp.fallback[base + __popc(mask & ((1u << lane) - 1))] = c;
        }
    }
}

// The stiff kinetics of one queued cell whose recovered state is stored.
template <int NS, class Rt>
__device__ __forceinline__ void react_queued(const DevMech &m, const DevState &st, long long n3, long long c,
                                             double dtm, int max_substeps, int counter)
{
    CellState<NS> cell;
    load_recovered<NS>(st, n3, c, cell);
    count_threads(&st.counters[counter]);
    ThermoCache<NS> tcache;
    if (react_or_defer<NS, Rt>(m, st, n3, c, cell, dtm, max_substeps, tcache))
        store_cell<NS>(m, st, n3, c, cell, &tcache);
}

// Position `pos` of the batch's queues taken end to end: the instance holding
// it and the position within that instance's queue (lengths from len(q)).
template <class Len>
__device__ __forceinline__ int batch_locate(int n, int pos, Len len, int &local)
{
    int q = 0, off = 0;
    for (; q < n; ++q) {
        const int l = len(q);
        if (pos < off + l)
            break;
        off += l;
    }
    local = pos - off;
    return q;
}

// The stiff-fallback queues of every instance of a batch drained by one fixed
// grid: warps take 32 positions at a time from one counter over the queues
// taken end to end (the shared reacting-cell work queue), so the cells of all
// instances are spread over the whole GPU. Per cell the same work as
// k_react_queue; every instance's statistics go to its own counters.
template <int NS, class Rt>
__global__ void __launch_bounds__(128) k_react_queue_batch(const __grid_constant__ DevMech m,
                                                           const BatchCell *__restrict__ tab, int n, int *next,
                                                           int max_substeps, int counter)
{
    auto len = [&](int q) { return tab[q].count ? *(volatile const int *)tab[q].count : 0; };
    int total = 0;
    for (int q = 0; q < n; ++q) total += len(q);
    if (total == 0)
        return;
    const int lane = threadIdx.x & 31;
    for (;;) {
        int base = 0;
        if (lane == 0)
            base = atomicAdd(next, 32);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= total)
            break;
        const int pos = base + lane;
        if (pos < total) {
            int local = 0;
            const int q = batch_locate(n, pos, len, local);
            if (q < n) {
                const BatchCell &b = tab[q];
                react_queued<NS, Rt>(m, b.st, b.n3, b.queue[local], *b.dt, max_substeps, counter);
            }
        }
    }
}

// The stiff kinetics on a queue of cells whose recovered state is stored.
template <int NS, class Rt>
__global__ void __launch_bounds__(128) k_react_queue(const __grid_constant__ DevMech m, const DevGrid g,
                                                     const DevState st, const int *__restrict__ queue, int *count,
                                                     const double *__restrict__ dt_dev, int max_substeps, int counter)
{
    // A fixed grid drains the queue (its length is read on the device): each
    // warp takes the next 32 cells from count[1] (reset before the launch).
    const int nq = *(volatile int *)count;
    if (nq == 0) // an empty queue: no warp touches the shared counter
        return;
    const int lane = threadIdx.x & 31;
    int *next = count + 1;
    for (;;) {
        int base = 0;
        if (lane == 0)
            base = atomicAdd(next, 32);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= nq)
            break;
        const int q = base + lane;
        if (q < nq)
            react_queued<NS, Rt>(m, st, g.n3, queue[q], *dt_dev, max_substeps, counter);
    }
}

// Nchem routing of the learned mode: each active cell's Nchem is predicted
// (Reaction::TrapezoidPrediction, src/Reaction.cpp:865-942); a cell needing at
// most lp.min_nchem substeps takes the stiff kinetics here (its substeps cost
// less than the model's evaluation and carry no model error), the others are
// appended to the model's queue with their inputs (lp.queue, lp.feat, length
// lp.counts[0]). With
// lp.min_nchem <= 0 every active cell goes to the model unpredicted. A fixed
// grid drains the active queue (length lp.counts[3], warp grabs on counts[4]).
template <int NS, class Rt>
__global__ void __launch_bounds__(128) k_learned_route(const __grid_constant__ DevMech m, const DevGrid g,
                                                       const DevState st, LearnedParams lp,
                                                       const double *__restrict__ dt_dev, int max_substeps)
{
    const int nq = *(volatile int *)(lp.counts + 3);
    if (nq == 0)
        return;
    const int lane = threadIdx.x & 31;
    const long long n3 = g.n3;
    for (;;) {
        int base = 0;
        if (lane == 0)
            base = atomicAdd(lp.counts + 4, 32);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= nq)
            break;
        const int q = base + lane;
        bool to_model = false;
        long long c = 0;
        CellState<NS> cell;
        if (q < nq) {
            c = lp.active[q];
            to_model = true;
            load_recovered<NS>(st, n3, c, cell);
            if (lp.min_nchem > 0) {
                double mc[NS];
                SpeciesRates<NS> rates;
                const double dtm = *dt_dev;
                bool bad;
                const int nchem = predict_nchem<NS, Rt>(m, cell, dtm, max_substeps, bad, mc, rates);
                if (nchem <= lp.min_nchem) {
                    to_model = false;
                    if (st.heavy && nchem > kHeavyNchem) {
                        push_heavy(st.heavy, c);
                    } else {
                        count_nchem(st.counters, nchem, bad);
                        ThermoCache<NS> tcache;
                        run_substeps<NS, Rt>(m, cell, dtm, nchem, mc, rates, st.cms ? st.cms + c : nullptr, n3, tcache);
                        st.nchem[c] = nchem;
                        store_cell<NS>(m, st, n3, c, cell, &tcache);
                    }
                }
            }
        }
        const unsigned routed = __ballot_sync(0xffffffffu, q < nq && !to_model);
        if (routed && lane == __ffs(routed) - 1)
            atomicAdd(&st.counters[kCntRouted], (unsigned long long)__popc(routed));
        const unsigned mask = __ballot_sync(0xffffffffu, to_model);
        if (mask) {
            int at = 0;
            if (lane == __ffs(mask) - 1)
                at = atomicAdd(&lp.counts[0], __popc(mask));
            at = __shfl_sync(0xffffffffu, at, __ffs(mask) - 1);
            if (to_model) {
                at += __popc(mask & ((1u << lane) - 1));
                lp.queue[at] = int(c);
                learned_features<NS>(m, lp, at, cell, *dt_dev);
            }
        }
    }
}

// ------------------------------------------------- independent cell samples
// (training data for the learned model: the stiff chemistry on a batch of
// constant-volume, constant-energy cells, each with its own dt)

// Conserved state of cells at rest from (T, p, Y): FieldInitial's formulas
// (src/Flowfield.cpp:226-262). cs: NS + 4 planes of n; Y: NS planes of n.
template <int NS>
__global__ void k_state_from_tpy(const __grid_constant__ DevMech m, long long n, const double *__restrict__ T,
                                 const double *__restrict__ p, const double *__restrict__ Y, double *cs, double *E)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    double y[NS], inv_w = 0, e = 0;
#pragma unroll
    for (int s = 0; s < NS; ++s) y[s] = Y[s * n + i];
#pragma unroll
    for (int s = 0; s < NS; ++s) inv_w += y[s] / m.mw[s];
    const double Tc = T[i];
    const double D = p[i] / (kRUniv * 1000 * inv_w * Tc);
    const TPow pw = make_tpow(Tc, true);
#pragma unroll
    for (int s = 0; s < NS; ++s) e += y[s] * (h_species<NS>(m, pw, m.ri[s], s) - m.ri[s] * Tc);
#pragma unroll
    for (int s = 0; s < NS; ++s) cs[s * n + i] = D * y[s];
    cs[(NS + 0) * n + i] = 0;
    cs[(NS + 1) * n + i] = 0;
    cs[(NS + 2) * n + i] = 0;
    cs[(NS + 3) * n + i] = D * e * 1000;
    E[i] = e * 1000;
}

// A sample's state (planes of n values) and back.
template <int NS>
__device__ __forceinline__ void load_sample(long long n, long long i, const double *cs, const double *T, const double *E,
                                            CellState<NS> &cell)
{
#pragma unroll
    for (int q = 0; q < NS + 4; ++q) cell.cs[q] = cs[q * n + i];
    load_temperature<NS>(cell, T[i]);
    cell.E = E[i];
    double D = 0;
#pragma unroll
    for (int s = 0; s < NS; ++s) D += cell.cs[s];
#pragma unroll
    for (int s = 0; s < NS; ++s) cell.Y[s] = cell.cs[s] / D;
    cell.D = D;
    cell.U = cell.cs[NS] / D;
    cell.V = cell.cs[NS + 1] / D;
    cell.W = cell.cs[NS + 2] / D;
}

template <int NS>
__device__ __forceinline__ void store_sample(long long n, long long i, double *cs, double *T, double *E,
                                             const CellState<NS> &cell)
{
#pragma unroll
    for (int q = 0; q < NS + 4; ++q) cs[q * n + i] = cell.cs[q];
    T[i] = cell.T;
    E[i] = cell.E;
}

// One chemistry step of each sample with its own dt, in place; samples of a
// large Nchem are left to k_chem_heavy (heavy = {count, next, samples...}, null:
// every sample on its own thread).
template <int NS, class Rt>
__global__ void __launch_bounds__(128) k_chem_samples(const __grid_constant__ DevMech m, long long n, double *cs,
                                                      double *T, double *E, const double *__restrict__ dt,
                                                      int *nchem, int max_substeps, unsigned long long *counters,
                                                      int *heavy)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    CellState<NS> cell;
    load_sample<NS>(n, i, cs, T, E, cell);
    double mc[NS];
    SpeciesRates<NS> rates;
    bool bad;
    const int nc = predict_nchem<NS, Rt>(m, cell, dt[i], max_substeps, bad, mc, rates);
    if (heavy && nc > kHeavyNchem) {
        push_heavy(heavy, i);
        return;
    }
    count_nchem(counters, nc, bad);
    ThermoCache<NS> tcache;
    run_substeps<NS, Rt>(m, cell, dt[i], nc, mc, rates, nullptr, 0, tcache);
    if (nchem)
        nchem[i] = nc;
    store_sample<NS>(n, i, cs, T, E, cell);
}

// ------------------------------------------------- warp-per-cell kinetics

#include "eu3d_heavy.cuh"

// Derived output fields of Update_after_CS that the timestep does not keep
// (Wav, Rgas, Cp, C, Ma; src/Flowfield.cpp:1606-1616), from the stored state.
template <int NS>
__global__ void k_derived(const __grid_constant__ DevMech m, const DevGrid g, const DevState st, int which,
                          double *out)
{
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.n3)
        return;
    const long long n3 = g.n3;
    double inv_w = 0;
#pragma unroll
    for (int s = 0; s < NS; ++s) inv_w += st.prim[(kY0 + s) * n3 + c] / m.mw[s];
    const double Wav = 1.0 / inv_w;
    double v;
    if (which == 0) {
        v = Wav;
    } else if (which == 1) {
        v = kRUniv * 1000 / Wav;
    } else if (which == 2) {
        const TPow p = make_tpow(st.T[c], false);
        double cp = 0;
#pragma unroll
        for (int s = 0; s < NS; ++s) cp += cp_species<NS>(m, p, m.ri[s], s) * st.prim[(kY0 + s) * n3 + c];
        v = cp * 1000;
    } else {
        const double C = sqrt(st.prim[kG * n3 + c] * st.prim[kP * n3 + c] / st.prim[kD * n3 + c]);
        if (which == 3) {
            v = C;
        } else {
            const double U = st.prim[kU * n3 + c], V = st.prim[kV * n3 + c], W = st.prim[kW * n3 + c];
            v = sqrt(U * U + V * V + W * W) / C;
        }
    }
    out[c] = v;
}

// Stage combination of the three-stage TVD Runge-Kutta advection (Shu and
// Osher's SSP-RK3; the reference's TimeAdv::TVD_RK3, src/TimeAdv.cpp:210-221,
// is an empty stub): CS = a CS0 + b CS on the interior nodes, each product and
// the sum rounded separately (the same value in every arithmetic flavour).
__global__ void k_rk_combine(const DevGrid g, double *__restrict__ cs, const double *__restrict__ cs0, int planes,
                             double a, double b)
{
    const long long n = (long long)g.ni * g.nj * g.nk;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        interior_node(g, t, i, j, k);
        const long long c = cell_index(g, i, j, k);
        for (int q = 0; q < planes; ++q) {
            const long long o = q * g.n3 + c;
            cs[o] = __dadd_rn(__dmul_rn(a, cs0[o]), __dmul_rn(b, cs[o]));
        }
    }
}

// Writes a scalar (the timestep) into device memory from a kernel argument, so
// the value is captured at launch and the caller's copy may go away.
__global__ void k_set_value(double *dst, double v) { *dst = v; }

// Flowfield::CFLcondition (src/Flowfield.cpp:275-304): the smallest
// min(dx / (|u| + c), dy / (|v| + c)) over the interior nodes, c = sqrt(gamma p
// / rho), from the primitive planes the next flux step reads (FP32 in mixed
// precision). The spacings are the interior ones (the reference takes them
// from its first two ghost nodes, the same on a uniform grid with three or
// more nodes per axis). Positive doubles order as their bit patterns, so the
// block minima combine with an integer atomicMin into slot[0] (non-finite values
// map to the largest key and never win). The last block to arrive (the ticket in
// slot[1]) sets dt = cfl times the minimum, which the step's kernels read at
// *dt_dev, adds it to *time and resets the slot for the next step.
__global__ void __launch_bounds__(256) k_cfl(const DevGrid g, const DevState st, unsigned long long *slot, double cfl,
                                             double *dt_dev, double *time)
{
    const long long ncell = (long long)g.ni * g.nj * g.nk;
    const double dx = g.x[g.bc + 1] - g.x[g.bc], dy = g.y[g.bc + 1] - g.y[g.bc];
    const long long n3 = g.n3;
    double m = __longlong_as_double(0x7ff0000000000000LL);
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < ncell;
         t += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        interior_node(g, t, i, j, k);
        const long long c = cell_index(g, i, j, k);
        double P, D, U, V, G;
        if (st.prim32) {
            P = st.prim32[kP * n3 + c];
            D = st.prim32[kD * n3 + c];
            U = st.prim32[kU * n3 + c];
            V = st.prim32[kV * n3 + c];
            G = st.prim32[kG * n3 + c];
        } else {
            P = st.prim[kP * n3 + c];
            D = st.prim[kD * n3 + c];
            U = st.prim[kU * n3 + c];
            V = st.prim[kV * n3 + c];
            G = st.prim[kG * n3 + c];
        }
        const double C = sqrt(G * P / D);
        const double q = fmin(dx / (fabs(U) + C), dy / (fabs(V) + C));
        m = (q < m || !(q == q)) ? q : m; // a NaN sticks
    }
    unsigned long long b = (unsigned long long)__double_as_longlong(m);
    if (!(m >= 0.0)) // NaN (or a negative spacing): the largest key
        b = ~0ULL;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long v = __shfl_xor_sync(0xffffffffu, b, o);
        b = v < b ? v : b;
    }
    __shared__ unsigned long long wmin[8];
    if ((threadIdx.x & 31) == 0)
        wmin[threadIdx.x >> 5] = b;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) b = wmin[w] < b ? wmin[w] : b;
        atomicMin(slot, b);
        __threadfence();
        unsigned *ticket = reinterpret_cast<unsigned *>(slot + 1);
        if (atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1) { // wraps to 0
            const double dt = cfl * __longlong_as_double((long long)atomicExch(slot, 0x7ff0000000000000ULL));
            *dt_dev = dt;
            *time += dt;
        }
    }
}

} // namespace EU3D_NS
} // namespace eu3d
