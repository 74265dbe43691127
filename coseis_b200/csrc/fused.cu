// Fused step kernel: one pass over the mesh computes a whole time step of
// sord/sord.f90:42-44 for steps whose field-I/O hooks allow it:
//
//   cell phase   strain (9 support-operator gradients, PML g memory),
//                potency / moment point injections, Hooke's law, 1/V
//                (stress.f90:133-355) and the elastic hourglass cell values
//                yy * hourglass_nc(hg1 u + dt hg2 v) (acceleration.f90:136-163)
//   node phase   divergence (diff_cn) with PML p memory, hourglass_cn,
//                viscous-only hourglass in the PML, force injections,
//                a = f * mr, and the leapfrog update of the NEXT step
//                v' = v + dt a, u' = u + dt v' (time_integration.f90:27-41)
//
// A block of the interior kernel owns a 31 x 7 column of output nodes (32 x 8
// cells including the -1 halo) and streams along l.  Node planes are staged
// raw (u, v, gam, coordinates) by cp.async into shared memory one plane ahead,
// then turned into a 3-plane ring of the per-node values the cells need:
// w = u + gam v, the hourglass input hg1 u + dt hg2 v, and the coordinates.
// Cell planes (stress, hourglass values, divergence brackets) sit in a 2-plane
// ring.  Two barriers per plane.  Cells on tile borders are computed by both
// neighbours (from identical inputs, so identically).
//
// Nodes with a PML cell or node around them are left to the shell's kernels
// (shell.cuh; fast arithmetic on general meshes: slab.cuh), on the same plan:
// the owner of a cell writes its PML g memory, which is double-buffered like
// v and u so no block reads a value another block has already advanced.  In
// reference order the operations of a cell are the same in both, so a cell
// computed by either is bit-identical.  Point sources are applied in all.
//
// Support-operator brackets: rectilinear meshes use the per-direction
// constants verified at setup; terrain meshes (x = x(j), y = y(k)) compute
// the two z-dependent directions per cell from 1-D x, y and the z plane;
// general meshes compute all three.  Each cell's brackets are evaluated
// once and shared by the cell's gradient and its eight corner nodes'
// divergence (stencil.cuh: cell_cn_brackets).
//
// That is the step in reference order and, on general meshes, in fast
// arithmetic; rectilinear and terrain meshes take k_modal (modal.cuh) there.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <utility>
#include <vector>

#include "inject.cuh"
#include "modes.cuh"
#include "pair.cuh"
#include "sord.cuh"
#include "stencil.cuh"

// SORD_FAST_PAIRED selects packed f32x2 evaluation (pair.cuh) of the
// interior kernel's independent stencils; 0 evaluates them one at a time.
// Both give bit-identical results.
#ifndef SORD_FAST_PAIRED
#define SORD_FAST_PAIRED 0
#endif

namespace sordgpu {

constexpr bool kPaired = SORD_FAST_PAIRED != 0;
constexpr int FJ = 32, FK = 8;                // cell tile = threads
constexpr int FNJ = FJ + 1, FNK = FK + 1;     // node region of a plane
constexpr int FOJ = FJ - 1, FOK = FK - 1;     // output nodes of a tile
constexpr int NPL = FNJ * FNK;                // 297 nodes per plane
constexpr int NCL = FJ * FK;                  // 256 cells per plane
constexpr int NTH = FJ * FK;

// Shared-memory layout.  Node planes: float4 groups per node,
//   group 0 = (w_x, w_y, w_z, coordinate 0), group 1 = (h_x, h_y, h_z,
//   coordinate 1), group 2 = (coordinate 2, -, -, -) on general meshes,
// with w = u + gam v and h = hg1 u + dt hg2 v; terrain meshes store z as
// coordinate 0, general meshes x, y, z.  Cell planes: float4 groups per cell,
//   0: s_xx s_yy s_zz s_yz   1: s_zx s_xy hA0   2: hA1 hA2   3: hA3 hB0 hB1
//   4: hB2 hB3 - -   5..8: (b0, b1) divergence brackets of terms 2g, 2g+1
//   9, 10: b2 of terms 0..7 (general meshes)
// where hA_iq = hourglass values of mode iq for components (x, y) and
// hB_iq the z component, so every packed pair is an aligned float2.
template <int GEOM>
struct Lay {
    static constexpr int NCOORD = GEOM == GEOM_RECT ? 0 : GEOM == GEOM_TERRAIN ? 1 : 3;
    static constexpr int RAWF = 7 + NCOORD;                   // staged plane: u(3) v(3) gam coords
    static constexpr int RAWSZ = (RAWF * NPL + 3) & ~3;        // floats, float4-aligned end
    static constexpr int NGN = GEOM == GEOM_GENERAL ? 3 : 2;  // float4 groups per node
    static constexpr int NDIR = GEOM == GEOM_RECT ? 0 : GEOM == GEOM_TERRAIN ? 2 : 3;
    static constexpr int NGC = GEOM == GEOM_RECT ? 5 : GEOM == GEOM_TERRAIN ? 9 : 11;  // float4 groups per cell
    static constexpr size_t bytes = sizeof(float) * (size_t)RAWSZ + sizeof(float4) * (size_t)(3 * NPL * NGN + 2 * NCL * NGC);
    // fast arithmetic: one cell plane (each node plane reads only the cells
    // above it), which holds, per reading node column q, that node's whole
    // force terms from the cell: (fu_x, fu_y, fu_z, fl_x) as float4 group q
    // and (fl_y, fl_z) as float2 in groups 4-5
    static constexpr int NGCR = 6;
    static constexpr size_t bytes_fm = sizeof(float) * (size_t)RAWSZ + sizeof(float4) * (size_t)(3 * NPL * NGN + NCL * NGCR);
};
// scalar field numbers of the node and cell groups
__host__ __device__ constexpr int nf_co(int c) { return c == 0 ? 3 : c == 1 ? 7 : 8; }
__host__ __device__ constexpr int cf_hg(int iq, int ic) { return ic < 2 ? 6 + 2 * iq + ic : 14 + iq; }
__host__ __device__ constexpr int cf_br(int a, int t) { return a < 2 ? 20 + 2 * t + a : 36 + t; }

__device__ __forceinline__ void bmax(unsigned* dst, float v) {
    unsigned b = __float_as_uint(v);
    if (v != v) b = 0x7fc00000u;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
    __shared__ unsigned s[32];
    const int t = threadIdx.x + blockDim.x * threadIdx.y;
    const int lane = t & 31, warp = t >> 5, nw = (blockDim.x * blockDim.y + 31) >> 5;
    __syncthreads();
    if (lane == 0) s[warp] = b;
    __syncthreads();
    if (warp == 0) {
        b = lane < nw ? s[lane] : 0u;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
        if (lane == 0 && b) atomicMax(dst, b);
    }
}
__device__ __forceinline__ float fmaxn(float m, float c) { return (c != c || c > m) ? c : m; }

// Mass, statistics, acceleration output and the folded leapfrog update of
// node q = (jn, kn, l) with force f (acceleration.f90:235-238,
// time_integration.f90:32-35).  A node on either plane of a double-node
// fault keeps its force: the rupture step adds the fault traction to it,
// divides by the mass and, when the step is folded, advances its v and u;
// the fold copies its v and u into the new buffers.
template <bool FM = false>
__device__ __forceinline__ void finish_node(const StepArgs& A, long long q, int jn, int kn, int l, float (&f)[3],
                                            float m, const float (&uv)[6], float dt, float& st_a, float& st_v,
                                            float& st_u) {
    const int fc = A.fax == 0 ? jn : A.fax == 1 ? kn : l;
    const bool fnode = A.fax >= 0 && (unsigned)(fc - A.firup) <= 1u;
    const float u0 = uv[0], u1 = uv[1], u2 = uv[2], v0 = uv[3], v1 = uv[4], v2 = uv[5];
    if (fnode) {
#pragma unroll
        for (int i = 0; i < 3; i++) A.fout[i][q] = f[i];
        if (A.stats) {
            st_v = fmaxn(st_v, v0 * v0 + v1 * v1 + v2 * v2);
            st_u = fmaxn(st_u, u0 * u0 + u1 * u1 + u2 * u2);
        }
        if (A.fold) {
            A.vout[0][q] = v0; A.uout[0][q] = u0;
            A.vout[1][q] = v1; A.uout[1][q] = u1;
            A.vout[2][q] = v2; A.uout[2][q] = u2;
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < 3; i++) f[i] = f[i] * m;
    if (A.stats) {
        st_a = fmaxn(st_a, f[0] * f[0] + f[1] * f[1] + f[2] * f[2]);
        st_v = fmaxn(st_v, v0 * v0 + v1 * v1 + v2 * v2);
        st_u = fmaxn(st_u, u0 * u0 + u1 * u1 + u2 * u2);
    }
    if (A.aout[0])
#pragma unroll
        for (int i = 0; i < 3; i++) A.aout[i][q] = f[i];
    if (A.fold) {
        float a, b;
        if (FM) {
            a = fmaf(dt, f[0], v0); b = fmaf(dt, a, u0); A.vout[0][q] = a; A.uout[0][q] = b;
            a = fmaf(dt, f[1], v1); b = fmaf(dt, a, u1); A.vout[1][q] = a; A.uout[1][q] = b;
            a = fmaf(dt, f[2], v2); b = fmaf(dt, a, u2); A.vout[2][q] = a; A.uout[2][q] = b;
        } else {
            a = v0 + dt * f[0]; b = u0 + dt * a; A.vout[0][q] = a; A.uout[0][q] = b;
            a = v1 + dt * f[1]; b = u1 + dt * a; A.vout[1][q] = a; A.uout[1][q] = b;
            a = v2 + dt * f[2]; b = u2 + dt * a; A.vout[2][q] = a; A.uout[2][q] = b;
        }
    }
}

__device__ __forceinline__ long long slab_idx(const Geom& g, int axis, int t, int ii, int j, int k, int l, int ic) {
    long long e0 = axis == 0 ? t : g.nm[0], e1 = axis == 1 ? t : g.nm[1], e2 = axis == 2 ? t : g.nm[2];
    long long a0 = axis == 0 ? ii : j - 1, a1 = axis == 1 ? ii : k - 1, a2 = axis == 2 ? ii : l - 1;
    return a0 + e0 * (a1 + e1 * a2) + (long long)ic * e0 * e1 * e2;
}

constexpr int SJ = 16, SK = 16;  // shell tile (cells = threads)

// Zero one cell of the fast-arithmetic cell plane of the shell (layout of
// LaySl: NGCF groups of ncl float4) in the pattern the cell phase writes it:
// group 1 holds float2 values at index tid, which a float4 store at tid would
// miss (and would clear two other cells' values instead).
__device__ __forceinline__ void zero_cell_fm(float4* sC, int tid, int ncl) {
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    sC[tid] = z;
    reinterpret_cast<float2*>(sC + ncl)[tid] = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 2; i < 14; i++) sC[i * ncl + tid] = z;
}

// Zero one cell of the interior kernel's fast-arithmetic cell plane (Lay:
// NGCR groups: four float4 groups, then four float2 arrays).
__device__ __forceinline__ void zero_cell_fr(float4* sC, int tid, int ncl) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
        sC[q * ncl + tid] = make_float4(0.f, 0.f, 0.f, 0.f);
        reinterpret_cast<float2*>(sC + 4 * ncl)[q * ncl + tid] = make_float2(0.f, 0.f);
    }
}

// Interior kernel: tiles of 31 x 7 nodes from (A.jf, A.kf), planes A.lf0..A.lf1,
// strictly inside the non-PML region, with no PML or boundary terms.
// FM (fast arithmetic, general meshes; k_modal has the others): fused
// multiply-adds, brackets scaled by h once per cell, divergence brackets
// taken as the negated gradient brackets; equal to the reference-order
// kernel in exact arithmetic, not bit for bit.
template <int GEOM, bool FM>
__global__ void __launch_bounds__(NTH, GEOM == GEOM_GENERAL ? 1 : 2) k_interior(StepArgs A) {
    using L = Lay<GEOM>;
    constexpr int NGN = L::NGN, NGC = L::NGC, NDIR = L::NDIR;
    extern __shared__ float4 sm4[];
    static_assert(!FM || GEOM == GEOM_GENERAL, "k_modal takes the other meshes in fast arithmetic");
    float* sR = reinterpret_cast<float*>(sm4);  // [RAWF][NPL] staged plane
    float4* sN = sm4 + L::RAWSZ / 4;            // [3 slots][NGN][NPL]
    float4* sC = sN + 3 * NGN * NPL;            // [2 slots][NGC][NCL]; fast arithmetic [NGCR][NCL]
#define RAW(f, i) sR[(f) * NPL + (i)]
    const Geom& g = A.g;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + FJ * ty;
    const int L0 = A.lf0 + blockIdx.z * A.segl;
    const int L1 = min(L0 + A.segl - 1, A.lf1);
    const int j0 = A.jf + blockIdx.x * FOJ, k0 = A.kf + blockIdx.y * FOK;
    const int J = j0 - 1 + tx, K = k0 - 1 + ty;      // this thread's cell column
    const int jn = j0 + tx, kn = k0 + ty;            // this thread's node column
    // the last tile of each row may be partial: its cells past (jend, kend)
    // are computed but feed no output node
    const bool outcol = tx < FOJ && ty < FOK && jn <= A.jend && kn <= A.kend;
    const bool cellcol = J >= g.i1cell[0] && J <= g.i2cell[0] && K >= g.i1cell[1] && K <= g.i2cell[1];
    const bool owncol = J >= j0 && J <= A.jend && K >= k0 && K <= A.kend;
    const float h = g.h, dt = g.dt;
    const unsigned long long nz = f2_pack(A.negzero, A.negzero);  // (-0.0, -0.0) from the host (pair.cuh)
    float st_a = 0.f, st_v = 0.f, st_u = 0.f, st_w = 0.f;
    // terrain meshes: this thread's cell column's x (j, j+1) and y (k, k+1)
    float txa = 0.f, txb = 0.f, tya = 0.f, tyb = 0.f;
    if (GEOM == GEOM_TERRAIN && cellcol) {
        txa = A.x1d[J - 1];
        txb = A.x1d[J];
        tya = A.y1d[K - 1];
        tyb = A.y1d[K];
    }

    // point sources of the step in this block's box (cells j0-1.., nodes
    // j0..); a block outside the box around all of them does not look, and
    // only cells inside it do
    __shared__ Inject lpot[kLocalInject], lmom[kLocalInject], lfrc[kLocalInject];
    __shared__ int lcnt[3];
    int npot = 0, nmom = 0, nfrc = 0;
    if (A.ibox[0] <= j0 + FOJ - 1 && A.ibox[3] >= j0 - 1 && A.ibox[1] <= k0 + FOK - 1 && A.ibox[4] >= k0 - 1 &&
        A.ibox[2] <= L1 && A.ibox[5] >= L0 - 1) {
        gather_inject(A.pot, lpot, &lcnt[0], g, j0 - 1, j0 + FOJ - 1, k0 - 1, k0 + FOK - 1, L0 - 1, L1);
        gather_inject(A.mom, lmom, &lcnt[1], g, j0 - 1, j0 + FOJ - 1, k0 - 1, k0 + FOK - 1, L0 - 1, L1);
        gather_inject(A.force, lfrc, &lcnt[2], g, j0, j0 + FOJ - 1, k0, k0 + FOK - 1, L0, L1);
        __syncthreads();
        npot = lcnt[0];
        nmom = lcnt[1];
        nfrc = lcnt[2];
    }
    const bool scol = (npot != 0 || nmom != 0) && J >= A.ibox[0] && J <= A.ibox[3] && K >= A.ibox[1] && K <= A.ibox[4];

    // ---------------------------------------------------------------- loads
    // stage node plane l (u, v, gam, coordinates) into sR asynchronously
    auto fetch = [&](int l) {
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const int n = tid + r * NTH;
            if (n < NPL) {
                const int nj = n % FNJ, nk = n / FNJ;
                const int j = j0 - 1 + nj, k = k0 - 1 + nk;
                const bool ok = j <= g.nm[0] && k <= g.nm[1] && l >= 1 && l <= g.nm[2];
                if (ok) {
                    const long long q = g.idx(j, k, l);
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        cp_async4(&RAW(c, n), A.uin[c] + q);
                        cp_async4(&RAW(3 + c, n), A.vin[c] + q);
                    }
                    cp_async4(&RAW(6, n), A.gam + q);
                    if (GEOM == GEOM_TERRAIN) cp_async4(&RAW(7, n), A.x[2] + q);
                    if (GEOM == GEOM_GENERAL)
#pragma unroll
                        for (int c = 0; c < 3; c++) cp_async4(&RAW(7 + c, n), A.x[c] + q);
                } else {
#pragma unroll
                    for (int f = 0; f < L::RAWF; f++) RAW(f, n) = 0.f;
                }
            }
        }
        cp_async_commit();
    };
    // staged plane -> ring slot: w1 = u + gam * v (time_integration.f90:36)
    // and the hourglass input hg1 u + dt hg2 v (acceleration.f90:141)
    auto store = [&](int slot) {
        float4* dst = sN + slot * (NGN * NPL);
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const int n = tid + r * NTH;
            if (n < NPL) {
                const float gm = RAW(6, n);
                float w[3], hh[3];
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const float u = RAW(c, n), v = RAW(3 + c, n);
                    w[c] = FM ? fmaf(gm, v, u) : u + gm * v;
                    hh[c] = FM ? fmaf(A.dh2, v, A.hg1 * u) : A.hg1 * u + A.dh2 * v;
                }
                const float c0 = L::NCOORD > 0 ? RAW(7, n) : 0.f;
                const float c1 = L::NCOORD > 1 ? RAW(8, n) : 0.f;
                dst[n] = make_float4(w[0], w[1], w[2], c0);
                dst[NPL + n] = make_float4(hh[0], hh[1], hh[2], c1);
                if (NGN > 2) dst[2 * NPL + n] = make_float4(L::NCOORD > 2 ? RAW(9, n) : 0.f, 0.f, 0.f, 0.f);
            }
        }
    };

    // per-plane statics of this thread's cell (lam, mu, 1/V, yy) and node
    // (mass ratio), loaded one plane ahead of their use
    float cur[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    auto stat_load = [&](int l, float* o) {
        const bool cv = cellcol && l >= g.i1cell[2] && l <= g.i2cell[2];
        const long long qc = cv ? g.idx(J, K, l) : 0;
        o[0] = cv ? A.lam[qc] : 0.f;
        o[1] = cv ? A.mu[qc] : 0.f;
        o[2] = cv ? A.vc[qc] : 0.f;
        o[3] = cv ? A.yy[qc] : 0.f;
        const bool nv = outcol && l >= g.i1node[2] && l <= g.i2node[2];
        o[4] = nv ? A.mr[g.idx(jn, kn, l)] : 0.f;
    };
    // this thread's node u, v (for the update and statistics), one plane ahead
    float uv[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    auto uv_load = [&](int l, float* o) {
        const bool nv = outcol && l >= g.i1node[2] && l <= g.i2node[2];
        const long long q = nv ? g.idx(jn, kn, l) : 0;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            o[c] = nv ? A.uin[c][q] : 0.f;
            o[3 + c] = nv ? A.vin[c][q] : 0.f;
        }
    };

    // one cell's results into cell slot cs (layout of Lay)
#define WRITE_CELL(cs, ed, eo, he, cnb)                                                                   \
    do {                                                                                                   \
        float4* cw_ = sC + (cs) * (NGC * NCL) + tid;                                                       \
        cw_[0] = make_float4(ed[0], ed[1], ed[2], eo[0]);                                                  \
        cw_[NCL] = make_float4(eo[1], eo[2], he[0], he[1]);                                                \
        cw_[2 * NCL] = make_float4(he[3], he[4], he[6], he[7]);                                            \
        cw_[3 * NCL] = make_float4(he[9], he[10], he[2], he[5]);                                           \
        cw_[4 * NCL] = make_float4(he[8], he[11], 0.f, 0.f);                                               \
        if (NDIR >= 2)                                                                                     \
            _Pragma("unroll") for (int q2 = 0; q2 < 4; q2++) cw_[(5 + q2) * NCL] =                         \
                make_float4(cnb[0][2 * q2], cnb[1][2 * q2], cnb[0][2 * q2 + 1], cnb[1][2 * q2 + 1]);        \
        if (NDIR == 3) {                                                                                   \
            cw_[9 * NCL] = make_float4(cnb[NDIR - 1][0], cnb[NDIR - 1][1], cnb[NDIR - 1][2], cnb[NDIR - 1][3]); \
            cw_[10 * NCL] = make_float4(cnb[NDIR - 1][4], cnb[NDIR - 1][5], cnb[NDIR - 1][6], cnb[NDIR - 1][7]); \
        }                                                                                                  \
    } while (0)

    // ---------------------------------------------------------------- cell phase
    // fast arithmetic: the terms of this thread's own cell for its own node
    // column (reader q = 0) stay in registers for the node phase
    float ownu[3] = {0.f, 0.f, 0.f}, ownl[3] = {0.f, 0.f, 0.f};
    auto cells = [&](int l) {
        const int cs = FM ? 0 : l & 1;
        if (!(l >= g.i1cell[2] && l <= g.i2cell[2])) {
            if constexpr (FM) {
                zero_cell_fr(sC, tid, NCL);
#pragma unroll
                for (int i = 0; i < 3; i++) { ownu[i] = 0.f; ownl[i] = 0.f; }
            } else {
                float4* cw = sC + cs * (NGC * NCL) + tid;
#pragma unroll
                for (int i = 0; i < NGC; i++) cw[i * NCL] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            return;
        }
        const long long q = g.idx(J, K, l);
        // corner values by corner id n = dj + 2 dk + 4 dl (node planes l, l+1)
        float Wc[3][8], Hc[3][8], X0[8], X1[8], X2[8];
        {
            const float4* p0 = sN + (l % 3) * (NGN * NPL) + (tx + FNJ * ty);
            const float4* p1 = sN + ((l + 1) % 3) * (NGN * NPL) + (tx + FNJ * ty);
#pragma unroll
            for (int n = 0; n < 8; n++) {
                const float4* p = ((n >> 2) ? p1 : p0) + (n & 1) + FNJ * ((n >> 1) & 1);
                const float4 a = p[0], b = p[NPL];
                Wc[0][n] = a.x; Wc[1][n] = a.y; Wc[2][n] = a.z;
                Hc[0][n] = b.x; Hc[1][n] = b.y; Hc[2][n] = b.z;
                if (GEOM == GEOM_TERRAIN) {
                    X0[n] = (n & 1) ? txb : txa;
                    X1[n] = ((n >> 1) & 1) ? tyb : tya;
                    X2[n] = a.w;
                } else if (GEOM == GEOM_GENERAL) {
                    X0[n] = a.w;
                    X1[n] = b.w;
                    X2[n] = p[2 * NPL].x;
                }
            }
        }
        // support-operator brackets; directions 0 and 1 in the two lanes
        float B[3][8];
        float cnb[NDIR > 0 ? NDIR : 1][8];
        if constexpr (FM) {
            // brackets scaled by h; divergence brackets = negated gradient brackets
            brackets_nc_g<float>(X1, X2, B[0]);
            brackets_nc_g<float>(X2, X0, B[1]);
            brackets_nc_g<float>(X0, X1, B[2]);
#pragma unroll
            for (int a = 0; a < 3; a++)
#pragma unroll
                for (int t = 0; t < 8; t++) B[a][t] = h * B[a][t];
#pragma unroll
            for (int a = 0; a < NDIR; a++)
#pragma unroll
                for (int t = 0; t < 8; t++) cnb[a][t] = -B[a][cn_of_nc(t)];
        } else if (GEOM == GEOM_RECT) {
#pragma unroll
            for (int a = 0; a < 3; a++)
#pragma unroll
                for (int t = 0; t < 8; t++) B[a][t] = A.br.bnc[a][t];
        } else if (kPaired) {
            F2 PB[8], PC[8], P[8], PN[8];
#pragma unroll
            for (int n = 0; n < 8; n++) {
                PB[n] = f2(X1[n], X2[n], nz);
                PC[n] = f2(X2[n], X0[n], nz);
            }
            brackets_nc_g<F2>(PB, PC, P);
            cell_cn_brackets_g<F2>(PB, PC, P, PN, f2(0.0f, nz));
#pragma unroll
            for (int t = 0; t < 8; t++) {
                B[0][t] = P[t].x();
                B[1][t] = P[t].y();
                cnb[0][t] = PN[t].x();
                cnb[1][t] = PN[t].y();
            }
            if (GEOM == GEOM_TERRAIN) {
#pragma unroll
                for (int t = 0; t < 8; t++) B[2][t] = A.br.bnc[2][t];
            } else {
                brackets_nc_g<float>(X0, X1, B[2]);
                cell_cn_brackets_g<float>(X0, X1, B[2], cnb[NDIR - 1], 0.0f);
            }
        } else {
            brackets_nc_g<float>(X1, X2, B[0]);
            cell_cn_brackets_g<float>(X1, X2, B[0], cnb[0], 0.0f);
            brackets_nc_g<float>(X2, X0, B[1]);
            cell_cn_brackets_g<float>(X2, X0, B[1], cnb[1], 0.0f);
            if (GEOM == GEOM_TERRAIN) {
#pragma unroll
                for (int t = 0; t < 8; t++) B[2][t] = A.br.bnc[2][t];
            } else {
                brackets_nc_g<float>(X0, X1, B[2]);
                cell_cn_brackets_g<float>(X0, X1, B[2], cnb[NDIR - 1], 0.0f);
            }
        }
        float ed[3], eo[3], he[12];
#pragma unroll
        for (int i = 0; i < 12; i++) he[i] = 0.f;
        const bool own = owncol && l >= L0;
        if constexpr (FM) {
            // gradients; the off-diagonal pairs are summed here and halved
            // with the modulus below
            float sg[3][3];
#pragma unroll
            for (int ic = 0; ic < 3; ic++) {
                float W[8];
#pragma unroll
                for (int t = 0; t < 8; t++) W[t] = Wc[ic][term_corner(t)];
#pragma unroll
                for (int id = 0; id < 3; id++) sg[ic][id] = dot8(W, B[id]);
            }
#pragma unroll
            for (int i = 0; i < 3; i++) ed[i] = sg[i][i];
            eo[0] = sg[1][2] + sg[2][1];
            eo[1] = sg[0][2] + sg[2][0];
            eo[2] = sg[0][1] + sg[1][0];
        } else if constexpr (!kPaired) {
#pragma unroll
            for (int ic = 0; ic < 3; ic++) {
                float W[8];
#pragma unroll
                for (int t = 0; t < 8; t++) W[t] = Wc[ic][term_corner(t)];
#pragma unroll
                for (int iid = 0; iid < 3; iid++) {
                    const int id = (ic + iid + 1) % 3;
                    const float s = stencil8(W, B[id], h);
                    if (ic == id) ed[ic] = s;
                    else if (ic < id) eo[3 - ic - id] = 0.5f * s;
                    else eo[3 - ic - id] = eo[3 - ic - id] + 0.5f * s;
                }
            }
        } else {
            // strain of an interior cell: s[ic][id] = stencil8(w_ic, B[id]);
            // (ic0, ic1) paired per iid, ic2's first two directions paired
            const F2 h2 = f2(h, nz);
            float sg[3][3];
            F2 W01[8];
            float W2v[8];
#pragma unroll
            for (int t = 0; t < 8; t++) {
                const int n = term_corner(t);
                W01[t] = f2(Wc[0][n], Wc[1][n], nz);
                W2v[t] = Wc[2][n];
            }
#pragma unroll
            for (int iid = 0; iid < 3; iid++) {
                const int ia = (0 + iid + 1) % 3, ib = (1 + iid + 1) % 3;
                F2 Bp[8];
#pragma unroll
                for (int t = 0; t < 8; t++) Bp[t] = f2(B[ia][t], B[ib][t], nz);
                const F2 r = stencil8<F2>(W01, Bp, h2);
                sg[0][ia] = r.x();
                sg[1][ib] = r.y();
            }
            {
                F2 W22[8], Bp[8];
#pragma unroll
                for (int t = 0; t < 8; t++) {
                    W22[t] = f2(W2v[t], nz);
                    Bp[t] = f2(B[0][t], B[1][t], nz);
                }
                const F2 r = stencil8<F2>(W22, Bp, h2);
                sg[2][0] = r.x();
                sg[2][1] = r.y();
                sg[2][2] = stencil8<float>(W2v, B[2], h);
            }
#pragma unroll
            for (int i = 0; i < 3; i++) ed[i] = sg[i][i];
            eo[0] = 0.5f * sg[1][2] + 0.5f * sg[2][1];
            eo[1] = 0.5f * sg[0][2] + 0.5f * sg[2][0];
            eo[2] = 0.5f * sg[0][1] + 0.5f * sg[1][0];
        }
        const bool src = scol && l >= A.ibox[2] && l <= A.ibox[5];
        if (src && npot != 0) {
            // strain (fast arithmetic carries the off-diagonal terms twice)
            float pd[3] = {0.f, 0.f, 0.f}, po[3] = {0.f, 0.f, 0.f};
            apply_inject(lpot, npot, A.pot, q, FM ? pd : ed, FM ? po : eo);
            if (FM)
#pragma unroll
                for (int i = 0; i < 3; i++) { ed[i] = ed[i] + pd[i]; eo[i] = fmaf(2.0f, po[i], eo[i]); }
        }
        if constexpr (FM) {
            // (2 mu e + lam tr e) / V; the off-diagonal sums carry the 1/2
            const float r = cur[2], mur = cur[1] * r, m2r = mur + mur;
            const float s1r = (cur[0] * r) * (ed[0] + ed[1] + ed[2]);
#pragma unroll
            for (int i = 0; i < 3; i++) { ed[i] = fmaf(m2r, ed[i], s1r); eo[i] = mur * eo[i]; }
            if (src && nmom != 0) {
                float pd[3] = {0.f, 0.f, 0.f}, po[3] = {0.f, 0.f, 0.f};
                apply_inject(lmom, nmom, A.mom, q, pd, po);
#pragma unroll
                for (int i = 0; i < 3; i++) { ed[i] = fmaf(pd[i], r, ed[i]); eo[i] = fmaf(po[i], r, eo[i]); }
            }
        } else {
            {
                const float lm = cur[0], m2 = 2.0f * cur[1];
                const float s1v = lm * (ed[0] + ed[1] + ed[2]);
#pragma unroll
                for (int i = 0; i < 3; i++) { ed[i] = m2 * ed[i] + s1v; eo[i] = m2 * eo[i]; }
            }
            if (src) apply_inject(lmom, nmom, A.mom, q, ed, eo);
            {
                const float r = cur[2];
#pragma unroll
                for (int i = 0; i < 3; i++) { ed[i] = ed[i] * r; eo[i] = eo[i] * r; }
            }
        }
        if (A.stats && own)
            st_w = fmaxn(st_w, (ed[0] * ed[0] + ed[1] * ed[1] + ed[2] * ed[2]) + 2.0f * (eo[0] * eo[0] + eo[1] * eo[1] + eo[2] * eo[2]));
        // elastic hourglass cell values (acceleration.f90:141-156)
        if (A.hourglass) {
            if constexpr (FM) {
                // the four mode sums by butterflies (stencil.cuh: hg_modes)
                const float y = cur[3];
#pragma unroll
                for (int ic = 0; ic < 3; ic++) {
                    float m[4];
                    hg_modes<float>(Hc[ic], m);
#pragma unroll
                    for (int iq = 0; iq < 4; iq++) he[3 * iq + ic] = m[iq] * y;
                }
            } else if constexpr (!kPaired) {
                const float y = cur[3];
#pragma unroll
                for (int ic = 0; ic < 3; ic++) {
                    float W2[8];
#pragma unroll
                    for (int t = 0; t < 8; t++) W2[t] = Hc[ic][hg_corner(t)];
#pragma unroll
                    for (int iq = 0; iq < 4; iq++) he[3 * iq + ic] = hg_sum(W2, iq) * y;
                }
            } else {
                const float y = cur[3];
                F2 H01[8];
                float H2v[8];
#pragma unroll
                for (int t = 0; t < 8; t++) {
                    const int n = hg_corner(t);
                    H01[t] = f2(Hc[0][n], Hc[1][n], nz);
                    H2v[t] = Hc[2][n];
                }
#pragma unroll
                for (int iq = 0; iq < 4; iq++) {
                    const F2 r = hg_sum<F2>(H01, iq) * f2(y, nz);
                    he[3 * iq] = r.x();
                    he[3 * iq + 1] = r.y();
                    he[3 * iq + 2] = hg_sum<float>(H2v, iq) * y;
                }
            }
        }
        if constexpr (FM) {
            // fast layout: for each node column q = cj + 2 ck that reads this
            // cell, the cell's whole terms of that column's force at node
            // plane l (fu, the node above the cell) and l + 1 (fl, the node
            // below it): the hourglass_cn sums (the signs of hourglass_cn
            // terms hg_term(7 - p) at cell position p, stencil.cuh:
            // hg_reader) plus the divergence of the cell's stress with that
            // node's diff_cn brackets
            const float S[6] = {ed[0], ed[1], ed[2], eo[0], eo[1], eo[2]};
            float hr[3][4];
#pragma unroll
            for (int ic = 0; ic < 3; ic++) {
                const float m[4] = {he[ic], he[3 + ic], he[6 + ic], he[9 + ic]};
                hg_readers_pre<float>(m, hr[ic]);
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int cj = q & 1, ck = q >> 1;
                const int tu = cj + 2 + 4 * ck, tl = cj + 4 * ck;
                float fu[3], fl[3];
#pragma unroll
                for (int ic = 0; ic < 3; ic++) hg_reader<float>(hr[ic], q, fu[ic], fl[ic]);
#pragma unroll
                for (int ic = 0; ic < 3; ic++)
#pragma unroll
                    for (int iid = 0; iid < 3; iid++) {
                        const int id = (ic + iid) % 3, comp = ic == id ? ic : 3 + (3 - ic - id);
                        fu[ic] = fmaf(S[comp], cnb[id][tu], fu[ic]);
                        fl[ic] = fmaf(S[comp], cnb[id][tl], fl[ic]);
                    }
                if (q == 0) {
#pragma unroll
                    for (int i = 0; i < 3; i++) { ownu[i] = fu[i]; ownl[i] = fl[i]; }
                    continue;
                }
                sC[q * NCL + tid] = make_float4(fu[0], fu[1], fu[2], fl[0]);
                reinterpret_cast<float2*>(sC + 4 * NCL)[q * NCL + tid] = make_float2(fl[1], fl[2]);
            }
        } else {
            WRITE_CELL(cs, ed, eo, he, cnb);
        }
    };

    // force sources at node q
    auto add_force = [&](long long q, float (&f)[3]) {
        if (nfrc == 0) return;
        const Inject* E = nfrc >= 0 ? lfrc : A.force.e;
        const int n = nfrc >= 0 ? nfrc : A.force.n;
        for (int e = 0; e < n; e++)
            if (E[e].idx == q) {
                const int c = E[e].comp;
                const float inc = E[e].inc;
                if (c == 0) f[0] = f[0] + inc;
                else if (c == 1) f[1] = f[1] + inc;
                else f[2] = f[2] + inc;
            }
    };

    // ---------------------------------------------------------------- node phase
    // The eight cells of node (jn, kn, l) are cell positions p = cj + 2 ck + 4 cl
    // at (J + cj, K + ck, l - 1 + cl); diff_cn term t sits at position
    // pt(t), hourglass_cn term t at position ph(t).
    // (reference order only; fast arithmetic uses nodes_fm below)
    auto nodes = [&](int l) {
        if (!outcol) return;
        const long long q = g.idx(jn, kn, l);
        const float4* c0 = sC + ((l - 1) & 1) * (NGC * NCL) + tid;  // cell plane l-1
        const float4* c1 = sC + (l & 1) * (NGC * NCL) + tid;        // cell plane l
        auto cpos = [&](int p) { return ((p >> 2) ? c1 : c0) + (p & 1) + FJ * ((p >> 1) & 1); };
        auto pt = [](int t) { return (t & 1) + 2 * (t >> 2) + 4 * ((t >> 1) & 1); };
        auto ph = [](int t) {
            const int o = hg_corner(t);
            return (1 - (o & 1)) + 2 * (1 - ((o >> 1) & 1)) + 4 * (1 - (o >> 2));
        };
        // stress (6) and divergence brackets by diff_cn term
        float S[6][8], Bc[3][8], HA0[2][8];  // HA0: mode-0 (x, y) hourglass values by diff_cn term
#pragma unroll
        for (int t = 0; t < 8; t++) {
            const float4* cp = cpos(pt(t));
            const float4 a = cp[0], b = cp[NCL];
            S[0][t] = a.x; S[1][t] = a.y; S[2][t] = a.z; S[3][t] = a.w; S[4][t] = b.x; S[5][t] = b.y;
            HA0[0][t] = b.z;
            HA0[1][t] = b.w;
            if (NDIR >= 2) {
                const float2 bb = reinterpret_cast<const float2*>(cp + (5 + t / 2) * NCL)[t % 2];
                Bc[0][t] = bb.x;
                Bc[1][t] = bb.y;
            }
            if (NDIR == 3) Bc[2][t] = reinterpret_cast<const float*>(cp + (9 + t / 4) * NCL)[t % 4];
            if (GEOM == GEOM_RECT)
#pragma unroll
                for (int id = 0; id < 3; id++) Bc[id][t] = A.br.bcn[id][t];
            if (GEOM == GEOM_TERRAIN) Bc[2][t] = A.br.bcn[2][t];
        }
        float f[3];
        if constexpr (!kPaired) {
#pragma unroll
            for (int ic = 0; ic < 3; ic++)
#pragma unroll
                for (int iid = 0; iid < 3; iid++) {
                    const int id = (ic + iid) % 3;
                    const int comp = ic == id ? ic : 3 + (3 - ic - id);
                    const float s = stencil8(S[comp], Bc[id], h);
                    f[ic] = iid == 0 ? s : f[ic] + s;
                }
        } else {
            // f[ic] = sum over iid of stencil8(sigma(ic, id), Bc[id]), id = (ic + iid) % 3;
            // (ic0, ic1) paired per iid, ic2's first two terms paired
            const F2 h2 = f2(h, nz);
            F2 f01;
#pragma unroll
            for (int iid = 0; iid < 3; iid++) {
                const int ia = iid, ib = (1 + iid) % 3;
                const int ca = 0 == ia ? 0 : 3 + (3 - 0 - ia), cb = 1 == ib ? 1 : 3 + (3 - 1 - ib);
                F2 Fp[8], Bp[8];
#pragma unroll
                for (int t = 0; t < 8; t++) {
                    Fp[t] = f2(S[ca][t], S[cb][t], nz);
                    Bp[t] = f2(Bc[ia][t], Bc[ib][t], nz);
                }
                const F2 r = stencil8<F2>(Fp, Bp, h2);
                f01 = iid == 0 ? r : f01 + r;
            }
            F2 Fp[8], Bp[8];
#pragma unroll
            for (int t = 0; t < 8; t++) {
                Fp[t] = f2(S[2][t], S[4][t], nz);
                Bp[t] = f2(Bc[2][t], Bc[0][t], nz);
            }
            const F2 r = stencil8<F2>(Fp, Bp, h2);
            f[2] = r.x() + r.y();
            f[2] = f[2] + stencil8<float>(S[3], Bc[1], h);
            f[0] = f01.x();
            f[1] = f01.y();
        }
        if (A.hourglass) {
            // hourglass values of mode iq by hourglass_cn term: (x, y) pair and z
#define HVALS(iq, hA, hB)                                                      \
    _Pragma("unroll") for (int t = 0; t < 8; t++) {                            \
        const float4* cp_ = cpos(ph(t));                                       \
        if ((iq) == 0) {                                                       \
            const float4 b_ = cp_[NCL];                                        \
            hA[t] = f2(b_.z, b_.w, nz);                                        \
            hB[t] = cp_[3 * NCL].z;                                            \
        } else if ((iq) == 1) {                                                \
            const float4 b_ = cp_[2 * NCL];                                    \
            hA[t] = f2(b_.x, b_.y, nz);                                        \
            hB[t] = cp_[3 * NCL].w;                                            \
        } else if ((iq) == 2) {                                                \
            const float4 b_ = cp_[2 * NCL];                                    \
            hA[t] = f2(b_.z, b_.w, nz);                                        \
            hB[t] = cp_[4 * NCL].x;                                            \
        } else {                                                               \
            const float4 b_ = cp_[3 * NCL];                                    \
            hA[t] = f2(b_.x, b_.y, nz);                                        \
            hB[t] = cp_[4 * NCL].y;                                            \
        }                                                                      \
    }
            if constexpr (!kPaired) {
                // each cell's hourglass groups once, as 128 / 64-bit loads:
                // g1.zw = mode 0 (x, y), g2 = modes 1, 2 (x, y), g3 = mode 3
                // (x, y), z of modes 0, 1, g4 = z of modes 2, 3
                float H[4][3][8];
#pragma unroll
                for (int t = 0; t < 8; t++) {
                    const int p = ph(t);
                    // diff_cn term at the same cell position
                    const int tp = (p & 1) + 4 * ((p >> 1) & 1) + 2 * (p >> 2);
                    const float4* cp_ = cpos(p);
                    const float4 g2 = cp_[2 * NCL], g3 = cp_[3 * NCL];
                    const float2 g4 = reinterpret_cast<const float2*>(cp_ + 4 * NCL)[0];
                    H[0][0][t] = HA0[0][tp]; H[0][1][t] = HA0[1][tp]; H[0][2][t] = g3.z;
                    H[1][0][t] = g2.x; H[1][1][t] = g2.y; H[1][2][t] = g3.w;
                    H[2][0][t] = g2.z; H[2][1][t] = g2.w; H[2][2][t] = g4.x;
                    H[3][0][t] = g3.x; H[3][1][t] = g3.y; H[3][2][t] = g4.y;
                }
#pragma unroll
                for (int iq = 0; iq < 4; iq++)
#pragma unroll
                    for (int ic = 0; ic < 3; ic++) f[ic] = f[ic] - hg_sum(H[iq][ic], iq);
            } else {
                F2 f01 = f2(f[0], f[1], nz);
#pragma unroll
                for (int iq = 0; iq < 4; iq++) {
                    F2 hA[8];
                    float hB[8];
                    HVALS(iq, hA, hB);
                    f01 = f01 - hg_sum<F2>(hA, iq);
                    f[2] = f[2] - hg_sum<float>(hB, iq);
                }
                f[0] = f01.x();
                f[1] = f01.y();
            }
        }
        add_force(q, f);
        finish_node<FM>(A, q, jn, kn, l, f, cur[4], uv, dt, st_a, st_v, st_u);
    };

    // ------------------------------------------------- node phase, fast arithmetic
    // Each cell plane is read once: at node plane l a thread takes the four
    // cells of plane l around its node column, adds their terms to node l
    // (cells above it) and keeps their terms for node l + 1 (cells below it)
    // in fc for the next plane.
    float fc[3] = {0.f, 0.f, 0.f};
    auto nodes_fm = [&](int l, bool finish) {
        if (!outcol) return;
        // the four cells of plane l around the node column: their terms for
        // node l (above them) and for node l + 1 (below), the latter carried
        // q = 0 is this thread's own cell, whose terms are in registers
        float fu[3] = {fc[0] + ownu[0], fc[1] + ownu[1], fc[2] + ownu[2]};
        float fl[3] = {ownl[0], ownl[1], ownl[2]};
#pragma unroll
        for (int q = 1; q < 4; q++) {
            const int ci = tid + (q & 1) + FJ * (q >> 1);  // the cell (J + cj, K + ck)
            const float4 a = sC[q * NCL + ci];
            const float2 b = reinterpret_cast<const float2*>(sC + 4 * NCL)[q * NCL + ci];
            fu[0] = fu[0] + a.x;
            fu[1] = fu[1] + a.y;
            fu[2] = fu[2] + a.z;
            fl[0] = fl[0] + a.w;
            fl[1] = fl[1] + b.x;
            fl[2] = fl[2] + b.y;
        }
#pragma unroll
        for (int i = 0; i < 3; i++) fc[i] = fl[i];
        if (!finish) return;
        add_force(g.idx(jn, kn, l), fu);
        finish_node<FM>(A, g.idx(jn, kn, l), jn, kn, l, fu, cur[4], uv, dt, st_a, st_v, st_u);
    };

    // ---------------------------------------------------------------- stream
    // ring: planes L0-1, L0, L0+1; staged: L0+2 in flight
#pragma unroll 1
    for (int p = -1; p <= 1; p++) {
        fetch(L0 + p);
        cp_async_wait_all();
        __syncthreads();
        store((L0 + p + 3) % 3);
        __syncthreads();
    }
    fetch(L0 + 2);
    stat_load(L0 - 1, cur);
    uv_load(L0, uv);
    // (one call of cells and of each node phase, so that all are inlined)
#pragma unroll 1
    for (int l = L0 - 1; l <= L1; l++) {
        const bool first = l < L0;  // the cell plane below the first node plane
        cells(l);
        float nxt[5], nuv[6];
        stat_load(l + 1, nxt);
        if (!first) cp_async_wait_all();
        __syncthreads();  // cell plane l complete, staged plane l+2 landed
        if (!first) store((l + 2) % 3);
        if constexpr (FM) nodes_fm(l, !first);
        else if (!first) nodes(l);
        if (!first) uv_load(l + 1, nuv);
        __syncthreads();  // ring slot l+2 complete, staging and cell slot l-1 free
        if (!first) {
            fetch(l + 3);
#pragma unroll
            for (int i = 0; i < 6; i++) uv[i] = nuv[i];
        }
#pragma unroll
        for (int i = 0; i < 5; i++) cur[i] = nxt[i];
    }
    cp_async_wait_all();
    if (A.stats) {
        bmax(A.red + 0, st_a);
        bmax(A.red + 1, st_v);
        bmax(A.red + 2, st_u);
        bmax(A.red + 3, st_w);
    }
#undef RAW
#undef WRITE_CELL
#undef HVALS
}

#include "modal.cuh"
#include "shell.cuh"
#include "slab.cuh"

// Arithmetic of the fused step.  The fast PML kernels give a cell or node one
// memory per axis, so a mesh on which the bands of opposite faces share cells
// (the front end refuses it, a deck need not) takes the kernels in reference
// order, which apply both, the near one first, as the reference does.
static int step_arith(const Solver& s) {
    for (int d = 0; d < 3; d++)
        if (s.g.npml > 0 && s.g.i2pml[d] - 1 <= s.g.i1pml[d]) return 0;
    return s.arith;
}

// Work decomposition of a fused step, fixed by the mesh.  The interior
// rectangle holds the node columns (j, k) whose adjacent cells all lie
// strictly inside the non-PML region, jf..jend x kf..kend; it is tiled by
// 31 x 7 node tiles from (jf, kf) (the last tile of a row may be partial)
// and runs the interior kernel over the node planes lf0..lf1 whose cells are
// interior (or the halo plane of a free surface).  Everything else -- the
// PML faces at full depth and the PML planes of the interior rectangle -- is
// covered by masked 15 x 15 node boxes for the shell kernel.  Boxes and tiles partition
// the nodes, so every node, and every PML memory, is updated once.
struct FusedPlan {
    bool ready = false;                         // all of it is there
    int jf = 0, jend = -1, kf = 0, kend = -1;   // interior rectangle (inclusive)
    int nbx = 0, nby = 0;                       // interior tiles
    int lf0 = 0, lf1 = -1;                      // interior node planes (inclusive)
    int segl = 0, nseg = 1;                     // interior planes per block, blocks per column
    // node boxes of the PML shell, six ints each (j0, k0, last j, last k,
    // first and last plane), by class of damped axes (MASK 1, 2, 4, 7)
    int nbox[4] = {0, 0, 0, 0};
    int* d_items = nullptr;
    // the PML-shell kernel runs on a second stream, concurrently with the
    // interior kernel (they write disjoint nodes and read the same inputs)
    cudaStream_t side = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    // each class of boxes on its own stream, forked from and joined back into
    // the stream of the shell launches, so that the classes' tails overlap
    cudaStream_t cst[4] = {};
    cudaEvent_t cfork = nullptr, cdone[4] = {};
};

static void plan_free(Solver& s, FusedPlan*& P) {
    if (!P) return;
    if (P->fork) cudaEventDestroy(P->fork);
    if (P->join) cudaEventDestroy(P->join);
    if (P->side) cudaStreamDestroy(P->side);
    if (P->cfork) cudaEventDestroy(P->cfork);
    for (int c = 0; c < 4; c++) {
        if (P->cdone[c]) cudaEventDestroy(P->cdone[c]);
        if (P->cst[c]) cudaStreamDestroy(P->cst[c]);
    }
    dev_free(s, P->d_items);
    delete P;
    P = nullptr;
}
void fused_free(Solver& s) {
    for (FusedPlan*& P : s.fplan) plan_free(s, P);
}

// Planes per block.  Each block streams its column through the planes, so
// a small mesh is cut into shorter plane ranges until both kernels have
// about kWaveBlocks blocks per SM; a range starts with a prologue of about
// two planes, so it is kept at kMinPlanes planes or more, and down to
// kFewPlanes only where the launch does not fill the chip: below a block per
// SM in fast arithmetic, below the two that fit in reference order, whose
// planes take longer.  61^3 nodes in reference order, 200 steps: eight
// planes 32.6 ms, four 27.5; one step of 24^3 275 and 250 us.  (Four below
// 592 blocks: 256 x 256 x 128 nodes 1 % slower; four below two blocks per SM
// in fast arithmetic: 203 x 149 x 97 nodes 2 % slower; three planes: no
// faster on 61^3.)
static constexpr int kItemPlanes = 96;
static constexpr int kMinPlanes = 8;
static constexpr int kFewPlanes = 4;
static constexpr int kWaveBlocks = 4;

// shell items covering node box [j1, j2] x [k1, k2] x [l1, l2], of at most
// ipl planes and as even as they can be: a launch lasts as long as its
// longest item
static void push_box(std::vector<int>& v, int ipl, int j1, int j2, int k1, int k2, int l1, int l2) {
    const int planes = l2 - l1 + 1, parts = (planes + ipl - 1) / ipl;
    ipl = parts > 0 ? (planes + parts - 1) / parts : 1;
    for (int a = l1; a <= l2; a += ipl)
        for (int k = k1; k <= k2; k += SK - 1)
            for (int j = j1; j <= j2; j += SJ - 1) {
                const int it[6] = {j, k, std::min(j2, j + SJ - 2), std::min(k2, k + SK - 2), a,
                                   std::min(l2, a + ipl - 1)};
                v.insert(v.end(), it, it + 6);
            }
}

static FusedPlan& fused_plan(Solver& s) {
    // one for each arithmetic, which may change between any two steps
    FusedPlan*& P = s.fplan[step_arith(s)];
    if (P && P->ready) return *P;
    plan_free(s, P);
    P = new FusedPlan();
    // shortest plane range of a launch that does not fill the chip
    const int few = kFewPlanes;
    const Geom& g = s.g;
    // Node c along axis d is interior when it is outside the PML and each
    // adjacent cell is either a real cell outside the PML or a cell outside
    // the mesh (a boundary without PML, whose coefficients are zero: the
    // kernel then adds exactly zero for it, as the reference does).
    auto cin = [&](int d, int c) { return c > g.i1pml[d] && c < g.i2pml[d] - 1 && c >= g.i1cell[d] && c <= g.i2cell[d]; };
    auto cellok = [&](int d, int c) { return c < g.i1cell[d] || c > g.i2cell[d] || cin(d, c); };
    auto nodeok = [&](int d, int c) { return c >= g.i1pml[d] + 1 && c <= g.i2pml[d] - 1 && cellok(d, c - 1) && cellok(d, c); };
    auto range = [&](int d, int& a, int& b) {
        a = 0;
        b = -1;
        for (int c = g.i1node[d]; c <= g.i2node[d]; c++)
            if (nodeok(d, c)) {
                if (b < a) a = c;
                if (b == c - 1 || b < a) b = c;
            }
    };
    range(0, P->jf, P->jend);
    range(1, P->kf, P->kend);
    range(2, P->lf0, P->lf1);
    const bool inner = P->jend >= P->jf && P->kend >= P->kf && P->lf1 >= P->lf0;
    const int L1 = g.i1node[2], L2 = g.i2node[2];
    int sms = 148;
    SORD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s.device));
    const int want = kWaveBlocks * sms;
    // regions of the shell, cut where the PML of another axis begins so that
    // each is damped along as few axes as possible (its class)
    struct RegionBox {
        int lo[3], hi[3];
    };
    std::vector<RegionBox> rb;
    auto add = [&](int j1, int j2, int k1, int k2, int l1, int l2) {
        if (j1 <= j2 && k1 <= k2 && l1 <= l2) rb.push_back({{j1, k1, l1}, {j2, k2, l2}});
    };
    if (!inner) {
        add(g.i1node[0], g.i2node[0], g.i1node[1], g.i2node[1], L1, L2);
    } else {
        const int kr[3][2] = {{g.i1node[1], P->kf - 1}, {P->kf, P->kend}, {P->kend + 1, g.i2node[1]}};
        const int lr[3][2] = {{L1, P->lf0 - 1}, {P->lf0, P->lf1}, {P->lf1 + 1, L2}};
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++) {
                add(g.i1node[0], P->jf - 1, kr[a][0], kr[a][1], lr[b][0], lr[b][1]);
                add(P->jend + 1, g.i2node[0], kr[a][0], kr[a][1], lr[b][0], lr[b][1]);
            }
        for (int b = 0; b < 3; b++) {
            add(P->jf, P->jend, g.i1node[1], P->kf - 1, lr[b][0], lr[b][1]);
            add(P->jf, P->jend, P->kend + 1, g.i2node[1], lr[b][0], lr[b][1]);
        }
        add(P->jf, P->jend, P->kf, P->kend, L1, P->lf0 - 1);
        add(P->jf, P->jend, P->kf, P->kend, P->lf1 + 1, L2);
    }
    // class of a node box: axis d needs the PML terms when a real cell
    // the box computes (node range a..b -> cells a-1..b) or one of its real
    // nodes lies in a PML slab of d; one axis -> its own class, more -> all
    auto klass = [&](const int* lo, const int* hi) {
        int m = 0;
        for (int d = 0; d < 3; d++) {
            for (int c = std::max(lo[d] - 1, g.i1cell[d]); c <= std::min(hi[d], g.i2cell[d]); c++)
                if (c <= g.i1pml[d] || c >= g.i2pml[d] - 1) m |= 1 << d;
            for (int c = std::max(lo[d], g.i1node[d]); c <= std::min(hi[d], g.i2node[d]); c++)
                if (c <= g.i1pml[d] || c >= g.i2pml[d]) m |= 1 << d;
        }
        return m == 2 ? 1 : m == 4 ? 2 : (m == 0 || m == 1) ? 0 : 3;
    };
    // Planes per item, per class: each class is one launch (on its own
    // stream), so its items are cut as long as the launch still has about
    // kWaveBlocks blocks per SM, and no shorter than kMinPlanes, or than
    // kFewPlanes where less is resident than could be.
    std::vector<int> rcls;
    for (const RegionBox& r : rb) rcls.push_back(klass(r.lo, r.hi));
    int iplc[4];
    for (int c = 0; c < 4; c++) {
        auto count = [&](int ipl) {
            long long n = 0;
            for (size_t i = 0; i < rb.size(); i++)
                if (rcls[i] == c)
                    n += (long long)((rb[i].hi[0] - rb[i].lo[0]) / (SJ - 1) + 1) * ((rb[i].hi[1] - rb[i].lo[1]) / (SK - 1) + 1) *
                         ((rb[i].hi[2] - rb[i].lo[2]) / ipl + 1);
            return n;
        };
        int ipl = kItemPlanes;
        while (ipl > kMinPlanes && count(ipl) < want) ipl = std::max(kMinPlanes, ipl * 2 / 3);
        while (ipl > few && count(ipl) < (step_arith(s) ? sms : 2 * sms)) ipl = std::max(few, ipl * 2 / 3);
        iplc[c] = ipl;
    }
    // boxes by their own class (a range of planes may miss the PML of z)
    std::vector<int> boxes, byclass[4];
    for (size_t i = 0; i < rb.size(); i++)
        push_box(boxes, iplc[rcls[i]], rb[i].lo[0], rb[i].hi[0], rb[i].lo[1], rb[i].hi[1], rb[i].lo[2], rb[i].hi[2]);
    for (size_t i = 0; i < boxes.size(); i += 6) {
        const int* b = &boxes[i];
        const int lo[3] = {b[0], b[1], b[4]}, hi[3] = {b[2], b[3], b[5]};
        std::vector<int>& v = byclass[klass(lo, hi)];
        v.insert(v.end(), b, b + 6);
    }
    std::vector<int> items;
    for (int c = 0; c < 4; c++) {
        P->nbox[c] = (int)byclass[c].size() / 6;
        items.insert(items.end(), byclass[c].begin(), byclass[c].end());
    }
    if (!inner) {
        P->jend = P->jf - 1;
    } else {
        P->nbx = (int)div_up(P->jend - P->jf + 1, FOJ);
        P->nby = (int)div_up(P->kend - P->kf + 1, FOK);
        const int planes = P->lf1 - P->lf0 + 1, cols = P->nbx * P->nby;
        // the split that takes the fewest plane times: rounds of two blocks
        // per SM, as many as are resident on rectilinear and terrain meshes
        // (one on general meshes, for which the rule has not been tuned), each
        // block its planes and a prologue of about two.  (An
        // even spread with half a last round, as if blocks did not come in
        // rounds, splits further: 5 % slower on 256 x 256 x 128 nodes in
        // reference order, where the shell's blocks fill the gaps anyway.)
        double best = 0;
        for (int n = 1; n <= std::max(1, planes / few); n++) {
            const int len = (planes + n - 1) / n;
            const long long blocks = (long long)cols * ((planes + len - 1) / len);
            const double t = (double)((blocks + 2 * sms - 1) / (2 * sms)) * (len + 2);
            if (n == 1 || t < best) {
                best = t;
                P->segl = len;
            }
        }
        P->nseg = (planes + P->segl - 1) / P->segl;
    }
    SORD_CUDA(dev_malloc(s, (void**)&P->d_items, sizeof(int) * std::max<size_t>(items.size(), 6)));
    if (!items.empty()) {
        SORD_CUDA(cudaMemcpyAsync(P->d_items, items.data(), sizeof(int) * items.size(), cudaMemcpyHostToDevice, s.stream));
        SORD_CUDA(cudaStreamSynchronize(s.stream));
    }
    SORD_CUDA(cudaEventCreateWithFlags(&P->fork, cudaEventDisableTiming));
    SORD_CUDA(cudaEventCreateWithFlags(&P->join, cudaEventDisableTiming));
    SORD_CUDA(cudaStreamCreateWithFlags(&P->side, cudaStreamNonBlocking));
    SORD_CUDA(cudaEventCreateWithFlags(&P->cfork, cudaEventDisableTiming));
    for (int c = 0; c < 4; c++) {
        SORD_CUDA(cudaEventCreateWithFlags(&P->cdone[c], cudaEventDisableTiming));
        SORD_CUDA(cudaStreamCreateWithFlags(&P->cst[c], cudaStreamNonBlocking));
    }
    P->ready = true;
    return *P;
}

template <int GEOM, int MASK>
static void launch_modal(Solver& s, const StepArgs& A, dim3 grid, cudaStream_t st) {
    using L = LayM<MASK>;
    if (A.fold && !A.stats && !A.aout[0] && A.fax < 0) {
        smem_limit((const void*)k_modal<GEOM, MASK, true>, (int)L::bytes);
        k_modal<GEOM, MASK, true><<<grid, dim3(L::TJ, L::TK), L::bytes, st>>>(A);
    } else {
        smem_limit((const void*)k_modal<GEOM, MASK, false>, (int)L::bytes);
        k_modal<GEOM, MASK, false><<<grid, dim3(L::TJ, L::TK), L::bytes, st>>>(A);
    }
    s.launches++;
    SORD_CUDA(cudaGetLastError());
}

// Mesh class of the step kernels: in fast arithmetic a rectilinear mesh
// whose cells are not boxes (a constant shear) takes the general kernels,
// since k_modal has the axes' own modes only.
static int step_class(const Solver& s) {
    if (!step_arith(s)) return s.geom;
    if (s.geom != GEOM_RECT) return s.geom;
    for (int a = 0; a < 3; a++) {
        double m[7] = {}, own = 0;
        for (int t = 0; t < 8; t++) {
            const int n = term_corner(t);
            const int x = (n & 1) * 2 - 1, y = ((n >> 1) & 1) * 2 - 1, z = (n >> 2) * 2 - 1;
            const int sg[7] = {x, y, z, x * y, y * z, x * z, x * y * z};
            for (int q = 0; q < 7; q++) m[q] += sg[q] * (double)s.br.bnc[a][t];
        }
        own = std::fabs(m[a]);
        for (int q = 0; q < 7; q++)
            if (q != a && std::fabs(m[q]) > 1e-6 * own) return GEOM_GENERAL;  // beyond FP32 rounding
    }
    return GEOM_RECT;
}

// Interior tiles.
template <int GEOM>
static void launch_interior(Solver& s, const StepArgs& A, dim3 grid, cudaStream_t st) {
    constexpr bool FM = GEOM == GEOM_GENERAL;  // fast arithmetic of the other meshes: k_modal
    if constexpr (!FM) {
        if (step_arith(s)) {
            launch_modal<GEOM, 0>(s, A, grid, st);
            return;
        }
    }
    const size_t bytes = FM && step_arith(s) ? Lay<GEOM>::bytes_fm : Lay<GEOM>::bytes;
    auto kern = FM && step_arith(s) ? k_interior<GEOM, FM> : k_interior<GEOM, false>;
    smem_limit((const void*)kern, (int)bytes);
    kern<<<grid, dim3(FJ, FK), bytes, st>>>(A);
    s.launches++;
    SORD_CUDA(cudaGetLastError());
}

// Do the fast kernels of a mesh class take its PML shell?  k_modal damps every
// node there by dt hg2, which the reference leaves out for a negative
// constant: k_shell then, beside k_modal's interior (300 x 150 x 150
// rectilinear: 504 us a step, general kernels throughout 840, reference order
// throughout 672).
static bool fast_shell(const Solver& s, int geom) {
    return step_arith(s) && (geom == GEOM_GENERAL || !(s.prm.hourglass[1] < 0.f));
}

// Boxes of the PML shell of one class.
template <int GEOM, int MASK>
static void launch_boxes(Solver& s, const StepArgs& A, unsigned n, cudaStream_t st) {
    if (fast_shell(s, GEOM)) {
        if constexpr (GEOM != GEOM_GENERAL) {
            launch_modal<GEOM, MASK>(s, A, dim3(n, 1, 1), st);
            return;
        } else {
            const size_t bytes = LaySl::bytes;
            smem_limit((const void*)k_slab<MASK>, (int)bytes);
            k_slab<MASK><<<dim3(n, 1, 1), dim3(SJ, SK), bytes, st>>>(A);
        }
    } else {
        const size_t bytes = LaySh<GEOM>::bytes;
        smem_limit((const void*)k_shell<GEOM, MASK>, (int)bytes);
        k_shell<GEOM, MASK><<<dim3(n, 1, 1), dim3(SJ, SK), bytes, st>>>(A);
    }
    s.launches++;
    SORD_CUDA(cudaGetLastError());
}

template <int GEOM>
static void launch_class(Solver& s, const StepArgs& A, int cls, unsigned n, cudaStream_t st) {
    if (cls == 0) launch_boxes<GEOM, 1>(s, A, n, st);
    else if (cls == 1) launch_boxes<GEOM, 2>(s, A, n, st);
    else if (cls == 2) launch_boxes<GEOM, 4>(s, A, n, st);
    else launch_boxes<GEOM, 7>(s, A, n, st);
}

// The statics of k_modal, laid out anew where they are not valid.
static const float4* modal_statics(Solver& s) {
    Device& d = s.d;
    float4* sta = (float4*)d.sd[0];
    if (!d.statics_valid) {
        k_statics<<<div_up(std::min(s.g.nv, 148LL * 64 * 256), 256), 256, 0, s.stream>>>(s.g, d.lam, d.mu, d.vc, d.yy, d.mr, sta);
        s.launches++;
        SORD_CUDA(cudaGetLastError());
        d.statics_there = d.statics_valid = true;
    }
    return sta;
}

void launch_fused(Solver& s, const InjectList& pot, const InjectList& mom, const InjectList& force,
                  const std::vector<Inject>& hpot, const std::vector<Inject>& hmom, const std::vector<Inject>& hforce,
                  bool fold, bool write_a, bool stats) {
    Device& d = s.d;
    FusedPlan& P = fused_plan(s);
    StepArgs A;
    A.g = s.g;
    A.br = s.br;
    for (int a = 0; a < 3; a++)
        for (int t = 0; t < 8; t++) {
            A.brh.bnc[a][t] = s.g.h * s.br.bnc[a][t];
            A.brh.bcn[a][t] = s.g.h * s.br.bcn[a][t];
        }
    for (int a = 0; a < 3; a++) {
        // the bracket's mode along its own axis: the mean over the corners of sign x bracket
        double m = 0;
        for (int t = 0; t < 8; t++) m += (((term_corner(t) >> a) & 1) * 2 - 1) * (double)A.brh.bnc[a][t];
        A.cm[a] = (float)(0.125 * m);
    }
    A.x1d = d.x1d;
    A.y1d = d.y1d;
    for (int i = 0; i < 3; i++) {
        A.x[i] = d.x[i];
        A.vin[i] = d.v[i];
        A.uin[i] = d.u[i];
        A.vout[i] = d.vb[i];
        A.uout[i] = d.ub[i];
        A.aout[i] = (write_a || !fold) ? d.w1n[i] : nullptr;
    }
    A.gam = d.gam; A.mr = d.mr; A.lam = d.lam; A.mu = d.mu; A.vc = d.vc; A.yy = d.yy;
    A.pmlc = d.pmlc;
    A.sl = d.slabs;
    for (int i = 0; i < 6; i++) A.gout[i] = d.gb[i];
    A.pot = pot; A.mom = mom; A.force = force;
    A.hourglass = (s.prm.hourglass[0] > 0.f || s.prm.hourglass[1] > 0.f) ? 1 : 0;
    A.hg1 = A.hourglass ? s.prm.hourglass[0] : 0.f;
    A.dh2 = A.hourglass ? s.g.dt * s.prm.hourglass[1] : 0.f;
    A.hgvisc = (s.prm.hourglass[1] > 0.f && s.g.npml > 0) ? 1 : 0;
    A.fold = fold ? 1 : 0;
    A.stats = stats ? 1 : 0;
    A.red = (unsigned*)d.red;
    A.jf = P.jf;
    A.kf = P.kf;
    A.jend = P.jend;
    A.kend = P.kend;
    A.lf0 = P.lf0;
    A.lf1 = P.lf1;
    A.segl = P.segl;
    A.items = P.d_items;
    A.negzero = -0.0f;
    A.fax = s.g.ifn - 1;
    A.firup = s.g.irup;
    for (int i = 0; i < 3; i++) A.fout[i] = d.w1n[i];

    int ib[6] = {INT_MAX, INT_MAX, INT_MAX, INT_MIN, INT_MIN, INT_MIN};
    for (const std::vector<Inject>* e : {&hpot, &hmom, &hforce})
        for (const Inject& x : *e) {
            const int c[3] = {(int)(x.idx % s.g.sy) + 1, (int)((x.idx / s.g.sy) % s.g.nm[1]) + 1, (int)(x.idx / s.g.sz) + 1};
            for (int d = 0; d < 3; d++) {
                ib[d] = std::min(ib[d], c[d]);
                ib[3 + d] = std::max(ib[3 + d], c[d]);
            }
        }
    for (int d = 0; d < 6; d++) A.ibox[d] = ib[d];

    const int geom = step_class(s);
    A.sta = step_arith(s) && geom != GEOM_GENERAL ? modal_statics(s) : nullptr;

    cudaEvent_t e0 = nullptr;
    s.prof_begin(KC_FUSED, &e0);
    const bool inner = P.nbx > 0 && P.nby > 0;
    const dim3 igrid(P.nbx, P.nby, P.nseg);
    // the shell: each class on its own stream
    auto shell_launches = [&](cudaStream_t st) {
        SORD_CUDA(cudaEventRecord(P.cfork, st));
        int off = 0;
        for (int m = 0; m < 4; m++) {
            if (P.nbox[m] == 0) continue;
            StepArgs B = A;
            B.items = P.d_items + 6 * (size_t)off;
            SORD_CUDA(cudaStreamWaitEvent(P.cst[m], P.cfork, 0));
            if (geom == GEOM_RECT) launch_class<GEOM_RECT>(s, B, m, (unsigned)P.nbox[m], P.cst[m]);
            else if (geom == GEOM_TERRAIN) launch_class<GEOM_TERRAIN>(s, B, m, (unsigned)P.nbox[m], P.cst[m]);
            else launch_class<GEOM_GENERAL>(s, B, m, (unsigned)P.nbox[m], P.cst[m]);
            SORD_CUDA(cudaEventRecord(P.cdone[m], P.cst[m]));
            SORD_CUDA(cudaStreamWaitEvent(st, P.cdone[m], 0));
            off += P.nbox[m];
        }
    };
    auto interior = [&]() {
        if (geom == GEOM_RECT) launch_interior<GEOM_RECT>(s, A, igrid, s.stream);
        else if (geom == GEOM_TERRAIN) launch_interior<GEOM_TERRAIN>(s, A, igrid, s.stream);
        else launch_interior<GEOM_GENERAL>(s, A, igrid, s.stream);
    };
    const bool shell = P.nbox[0] + P.nbox[1] + P.nbox[2] + P.nbox[3] > 0;
    if (inner && shell) {
        SORD_CUDA(cudaEventRecord(P.fork, s.stream));
        SORD_CUDA(cudaStreamWaitEvent(P.side, P.fork, 0));
        shell_launches(P.side);
        interior();
        SORD_CUDA(cudaEventRecord(P.join, P.side));
        SORD_CUDA(cudaStreamWaitEvent(s.stream, P.join, 0));
    } else if (inner) {
        interior();
    } else if (shell) {
        shell_launches(s.stream);
    }
    s.prof_end(KC_FUSED, e0);
    if (fold) {
        for (int i = 0; i < 3; i++) {
            std::swap(d.v[i], d.vb[i]);
            std::swap(d.u[i], d.ub[i]);
        }
    }
    for (int i = 0; i < 6; i++) std::swap(d.slabs.g[i], d.gb[i]);
}

}  // namespace sordgpu
