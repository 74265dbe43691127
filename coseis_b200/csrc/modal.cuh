// Step kernel in fast arithmetic on rectilinear and terrain meshes, interior
// and PML shell (included by fused.cu).
//
// The eight corners of a cell carry, along each axis, the sign -1 or +1, so
// every operator of the step is a short sum in the products of those signs
// (the modes j, k, l, jk, kl, jl, jkl of a corner field): the gradient of a
// field takes its modes j, k, l (and on a terrain mesh jk, kl, jl, with
// coefficients that are the z modes of the cell), the hourglass operator
// takes jk, kl, jl and jkl, and divergence and hourglass force put the
// cell's stress and hourglass values back on the corners with the same
// coefficients.  One pass of sums and differences therefore serves all
// gradients, and one serves the whole force.  Both split into a part within
// a node plane and a part across the two planes of a cell; the part within
// a plane is shared by the cells above and below it, so a thread that walks
// its cell column along l does it once per plane: it keeps the plane sums of
// w = u + gam v and of the hourglass input hg1 u + dt hg2 v of the last
// plane, and the force sums that the last cell leaves on its upper plane.
// A node plane's force reaches the nodes once both of its cells are in, as
// four corner values per thread, of which one is the thread's own node's.
//
// In the PML shell (MASK: the axes that may be damped in a box) a cell's
// gradient along a damped axis is that of v, through the g memory; along the
// others it is that of u, not w (stress.f90:18-131).  Divergence along a
// damped axis is kept apart until it reaches the node, which passes it
// through its p memory (acceleration.f90:37-104).  The hourglass force is
// split into its two parts: the viscous one, yy dt hg2 of v, acts on every
// node, the stiffness one, yy hg1 of u, only on nodes outside the PML
// (acceleration.f90:136-199), so it joins the force at the corner values.
//
// The interior is bound by instruction issue (0.71 of the slots on 203 x 149 x
// 97 terrain nodes); the shell's classes issue 0.33 to 0.46, their blocks
// waiting on the g and p memories.  Against the kernels that evaluated each
// bracket sum on its own, per launch on a B200:
//   512 x 512 x 256 terrain, 12-node PML  interior 1884 -> 1536 us, shell
//     classes x 415 -> 391, y 424 -> 327, z 288 -> 224, edges 162 -> 102 us
//   300 x 150 x 150 rectilinear, 10-node PML  interior 162 -> 134 us, x 65 ->
//     40, y 148 -> 88, z 97 -> 68, edges 99 -> 71 us
// The point sources are applied here: a separate launch for the boxes that
// hold them took 125 us of a 257 us step of 96 x 80 x 72 nodes, its 12
// blocks walking their planes alone.  Two cell columns per thread in packed
// f32x2 registers halve the arithmetic instructions but leave 12 warps per
// SM for chains twice as long: 153 us where one column per thread takes 77
// (203 x 149 x 97 terrain, interior).
#pragma once

// Tile of a block: TJ x TK cells, one per thread, (TJ - 1) x (TK - 1) output
// nodes.  The interior takes 32 x 8 (long rows: whole sectors), the shell
// 16 x 16 (slabs are 8 to 20 nodes thick along j or k).
template <int MASK>
struct LayM {
    static constexpr int TJ = MASK ? SJ : FJ, TK = MASK ? SK : FK;
    static constexpr int NJ = TJ + 1;        // nodes along j
    static constexpr int NP = NJ * (TK + 1);  // nodes per plane
    static constexpr int NT = TJ * TK;        // threads, cells per plane
    static constexpr int NS = 5;              // ring slots (node planes), each [(u, gam)][NP], [(v, z)][NP]
    static constexpr int ND = (MASK & 1) + ((MASK >> 1) & 1) + ((MASK >> 2) & 1);  // damped axes
    static constexpr int NSET = 1 + ND;  // force sets: the undamped part, then each damped axis's divergence
    // buffers of the force values: two save a barrier per plane.  (The edges
    // and corners have one, 95 KB a block instead of 144; a second block would
    // fit beside it, but their registers leave room for one only.)
    static constexpr int NB = MASK == 7 ? 1 : 2;
    static constexpr size_t bytes = 16 * (size_t)(NS * 2 * NP + NB * NSET * 3 * NT);
};

// What k_modal reads of cell (j, k, l) and node (j + 1, k + 1, l): lam / V,
// mu / V, yy and mr, zero off the mesh.
__global__ void k_statics(Geom g, const float* __restrict__ lam, const float* __restrict__ mu, const float* __restrict__ vc,
                          const float* __restrict__ yy, const float* __restrict__ mr, float4* __restrict__ out) {
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < g.nv; q += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(q % g.sy) + 1, k = (int)((q / g.sy) % g.nm[1]) + 1, l = (int)(q / g.sz) + 1;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        if (j >= g.i1cell[0] && j <= g.i2cell[0] && k >= g.i1cell[1] && k <= g.i2cell[1] && l >= g.i1cell[2] &&
            l <= g.i2cell[2]) {
            s.x = lam[q] * vc[q];
            s.y = mu[q] * vc[q];
            s.z = yy[q];
        }
        if (j + 1 >= g.i1node[0] && j + 1 <= g.i2node[0] && k + 1 >= g.i1node[1] && k + 1 <= g.i2node[1] &&
            l >= g.i1node[2] && l <= g.i2node[2])
            s.w = mr[q + 1 + g.sy];
        out[q] = s;
    }
}

// MASK 0: tiles of 31 x 7 nodes from (A.jf, A.kf), planes A.lf0..A.lf1,
// strictly inside the non-PML region.  Otherwise: the boxes A.items.
// Two cell planes are kept in flight (five ring slots) and the PML memories
// are read at the start of a plane's work.  Two blocks per SM leave a thread
// 128 registers: the interior fits, the classes of one axis spill (20 to 60
// bytes stored on rectilinear meshes, 120 to 330 on terrain); the edges and
// corners (MASK 7), whose memories of three axes are 18 values, take 199 to
// 244 registers for one block per SM (102 us against 137 with two, at 512 x
// 512 x 256).
// PLAIN: a folded step without statistics, acceleration output or fault,
// whose branches are compiled out.
template <int GEOM, int MASK, bool PLAIN>
__global__ void __launch_bounds__(LayM<MASK>::NT, MASK == 7 ? 1 : 2) k_modal(StepArgs A) {
    using L = LayM<MASK>;
    constexpr int TJ = L::TJ, TK = L::TK, NJ = L::NJ, NP = L::NP, NT = L::NT, NSET = L::NSET;
    constexpr bool TER = GEOM == GEOM_TERRAIN, PML = MASK != 0;
    constexpr bool DD[3] = {(MASK & 1) != 0, (MASK & 2) != 0, (MASK & 4) != 0};
    // the force set of each axis's divergence
    constexpr int SET[3] = {DD[0] ? 1 : 0, DD[1] ? (DD[0] ? 2 : 1) : 0, DD[2] ? L::ND : 0};
    constexpr bool hasl = !(MASK & 4) || (TER && (MASK & 3) != 3);  // the undamped set has a constant part
    extern __shared__ float4 sm4[];
    float4* sN = sm4;                  // [NS][2][NP] nodes
    float4* sX = sN + L::NS * 2 * NP;  // [NB][NSET][3][NT] force at corners (0,0) (1,0) (0,1)
    const Geom& g = A.g;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + TJ * ty;
    int j0, k0, jm, km, L0, L1;
    if constexpr (PML) {
        const int* it = A.items + 6 * blockIdx.x;
        j0 = it[0]; k0 = it[1]; jm = it[2]; km = it[3]; L0 = it[4]; L1 = it[5];
    } else {
        L0 = A.lf0 + blockIdx.z * A.segl;
        L1 = min(L0 + A.segl - 1, A.lf1);
        j0 = A.jf + blockIdx.x * (TJ - 1);
        k0 = A.kf + blockIdx.y * (TK - 1);
        jm = min(j0 + TJ - 2, A.jend);
        km = min(k0 + TK - 2, A.kend);
    }
    // point sources of the step in this block's box (cells j0-1.., nodes
    // j0..); a block outside the box around all of them does not look.  (A
    // block that took the sources of the tiles past its own too had every
    // cell walk them in every plane: 1171 us a step of 256 x 256 x 128 terrain
    // with four sources far apart, now 513, with one source 447.)
    __shared__ Inject lpot[kLocalInject], lmom[kLocalInject], lfrc[kLocalInject];
    __shared__ int lcnt[3];
    int npot = 0, nmom = 0, nfrc = 0;
    if (A.ibox[0] <= jm && A.ibox[3] >= j0 - 1 && A.ibox[1] <= km && A.ibox[4] >= k0 - 1 && A.ibox[2] <= L1 &&
        A.ibox[5] >= L0 - 1) {
        gather_inject(A.pot, lpot, &lcnt[0], g, j0 - 1, jm, k0 - 1, km, L0 - 1, L1);
        gather_inject(A.mom, lmom, &lcnt[1], g, j0 - 1, jm, k0 - 1, km, L0 - 1, L1);
        gather_inject(A.force, lfrc, &lcnt[2], g, j0, jm, k0, km, L0, L1);
        __syncthreads();
        npot = lcnt[0];
        nmom = lcnt[1];
        nfrc = lcnt[2];
    }
    const bool nsrc = npot != 0 || nmom != 0 || nfrc != 0;
    const int J = j0 - 1 + tx, K = k0 - 1 + ty;  // this thread's cell column
    const int jn = j0 + tx, kn = k0 + ty;        // its node column: corner (1, 1) of the cell column
    const bool outcol = tx < TJ - 1 && ty < TK - 1 && jn <= jm && kn <= km;
    const bool cellcol = J >= g.i1cell[0] && J <= g.i2cell[0] && K >= g.i1cell[1] && K <= g.i2cell[1];
    const bool owncol = cellcol && J >= j0 && J <= jm && K >= k0 && K <= km;
    float st_a = 0.f, st_v = 0.f, st_u = 0.f, st_w = 0.f;
    // coefficients of the modes: rectilinear, the gradient along each axis;
    // terrain, the factors of the z modes (3/4 and 1/4 of h dy for the
    // gradient along x, of h dx for y) and the constant gradient along z
    float cx = A.cm[0], cy = A.cm[1];
    if (TER) {
        cx = cellcol ? 0.25f * g.h * (A.y1d[K] - A.y1d[K - 1]) : 0.f;
        cy = cellcol ? 0.25f * g.h * (A.x1d[J] - A.x1d[J - 1]) : 0.f;
    }

    // ---------------------------------------------------------------- loads
    // the node copies of this thread as offsets in a plane; past the mesh
    // the last node or plane is copied instead: only cells off the mesh,
    // whose statics are zero, and cells that feed no output read it
    constexpr int NR = (NP + NT - 1) / NT;
    unsigned goff[NR];
#pragma unroll
    for (int r = 0; r < NR; r++) {
        const int n = tid + r * NT;
        const int j = min(j0 - 1 + n % NJ, g.nm[0]), k = min(k0 - 1 + n / NJ, g.nm[1]);
        goff[r] = (unsigned)(j - 1) + (unsigned)g.sy * (unsigned)(k - 1);
    }
    auto fetch = [&](int l, int slot) {
        if (l > L1 + 1) return;
        const long long pl = g.sz * (long long)(min(max(l, 1), g.nm[2]) - 1);
#pragma unroll
        for (int r = 0; r < NR; r++) {
            if ((r + 1) * NT > NP && tid + r * NT >= NP) continue;
            float* d = reinterpret_cast<float*>(sN + slot * (2 * NP) + tid + r * NT);
            const long long q = pl + goff[r];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                cp_async4(d + c, A.uin[c] + q);
                cp_async4(d + 4 * NP + c, A.vin[c] + q);
            }
            cp_async4(d + 3, A.gam + q);
            if (TER) cp_async4(d + 4 * NP + 3, A.x[2] + q);
        }
    };
    // per-plane statics (lam / V, mu / V, yy of the cell, mr of the node),
    // read one plane ahead: one 128-bit load
    const long long qcol = (long long)(J - 1) + g.sy * (long long)(K - 1);
    const long long qnod = qcol + 1 + g.sy;
    const bool incol = J <= g.nm[0] && K <= g.nm[1];
    auto stat_load = [&](int l) {
        return incol && l >= 1 && l <= L1 ? __ldg(A.sta + g.sz * (long long)(l - 1) + qcol)
                                          : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    // PML slab of cell c (memory g) or node c (memory p) along axis d: the
    // slab number (-1 outside), its layer and the 1-based damping index
    auto slab_of = [&](int d, int c, bool node, int& layer, int& p) {
        if (c <= g.i1pml[d]) {
            layer = c - (node ? g.i1node[d] : g.i1cell[d]);
            p = c + g.nnoff[d];
            return d;
        }
        if (c >= g.i2pml[d] - (node ? 0 : 1)) {
            layer = (node ? g.i2node[d] : g.i2cell[d]) - c;
            p = g.nn[d] - c - g.nnoff[d] + (node ? 1 : 0);
            return 3 + d;
        }
        return -1;
    };
    bool cold = false;  // the column is damped along j or k
    if constexpr (PML) {
        int a, p;
        if (DD[0]) cold = cold || slab_of(0, J, false, a, p) >= 0;
        if (DD[1]) cold = cold || slab_of(1, K, false, a, p) >= 0;
    }
    auto plane_damped = [&](int l) { return DD[2] && (l <= g.i1pml[2] || l >= g.i2pml[2] - 1); };

    // ------------------------------------------------------ plane sums
    // of the four nodes around the thread's column: (const, j, k, jk) of w;
    // interior: (j, k, jk) of the hourglass input hg1 u + dt hg2 v; shell:
    // (j, k, jk) of u and (const, j, k, jk) of v; z and minus its (j, k, jk)
    M3 w0[4], h0[3], v0[4], w1[4], h1[3], v1[4];
    float z0[4], zm0[3], z1[4], zm1[3];
    // damped: the cell plane that the sums are for lies in a PML slab of z
    auto gather = [&](int slot, bool damped, M3 (&w)[4], M3 (&h)[3], M3 (&v)[4], float (&z)[4], float (&zm)[3]) {
        const float4* p = sN + slot * (2 * NP) + tx + NJ * ty;
        M3 W[4], H[4], V[4];
        #pragma unroll
        for (int c = 0; c < 4; c++) {
            const float4 a = p[(c & 1) + NJ * (c >> 1)], b = p[NP + (c & 1) + NJ * (c >> 1)];
            const M3 u{a.x, a.y, a.z};
            V[c] = M3{b.x, b.y, b.z};
            // PML cells differentiate u instead of w
            const float gm = PML && (damped || cold) ? 0.f : a.w;
            // w = u + gam v (time_integration.f90:36) and hg1 u + dt hg2 v
            // (acceleration.f90:141)
            W[c] = m_fma(gm, V[c], u);
            H[c] = PML ? u : m_fma(A.dh2, V[c], A.hg1 * u);
            if (TER) z[c] = b.w;
        }
        m_sums4(W, w);
        m_sums3(H, h);
        if (PML) m_sums4(V, v);
        if (TER) {
            // differences of z first: z is large against them
            const float d0 = z[0] - z[1], d1 = z[2] - z[3];
            zm[0] = d0 + d1;
            zm[1] = (z[0] - z[2]) + (z[1] - z[3]);
            zm[2] = d1 - d0;
        }
    };

    // PML memory of this thread's cell (g) or node (p) of plane l along
    // axis d: the slab number (-1 outside the slabs), the element, the step
    // between components and the damping index
    auto mem_of = [&](int d, int l, bool node, long long& i, long long& step, int& p) {
        const bool in = node ? outcol && l >= L0 : cellcol && l >= g.i1cell[2] && l <= g.i2cell[2];
        if (!in) return -1;
        const int j = node ? jn : J, k = node ? kn : K;
        int layer;
        const int sb = slab_of(d, d == 0 ? j : d == 1 ? k : l, node, layer, p);
        if (sb < 0) return -1;
        const int t = node ? A.sl.tp[sb] : A.sl.tg[sb];
        i = slab_idx(g, d, t, layer, j, k, l, 0);
        step = slab_idx(g, d, t, layer, j, k, l, 1) - i;
        return sb;
    };
    auto mem_get = [&](int d, int l, bool node) {
        long long i, step;
        int p;
        const int sb = mem_of(d, l, node, i, step, p);
        if (sb < 0) return M3{0.f, 0.f, 0.f};
        const float* m = (node ? A.sl.p[sb] : A.sl.g[sb]) + i;
        return M3{m[0], m[step], m[2 * step]};
    };
    M3 gmem[3], pmem[3];  // those of plane l, read at the start of its work

    // ---------------------------------------------------------------- cells
    // acc: force sums (const, j, k, jk) that the last cell leaves on its
    // upper plane; T: those of plane l once cell l is in (per force set; q:
    // the stiffness hourglass of the shell).  The force is minus these sums.
    M3 acc[NSET][4], T[NSET][4], accq[4], Tq[4];
#pragma unroll
    for (int m = 0; m < 4; m++) {
#pragma unroll
        for (int s = 0; s < NSET; s++) acc[s][m] = M3{};
        accq[m] = M3{};
    }
    auto cell = [&](int l, const float4& st) {
        const float cz = A.cm[2];
        // terrain: coefficients of the gradients along x (p) and y (q); with
        // Z the z modes of the cell, d/dx = 3/4 dy (Zl j - Zj l) +
        // 1/4 dy (Zkl jk - Zjk kl), d/dy = 3/4 dx (Zl k - Zk l) +
        // 1/4 dx (Zjl jk - Zjk jl) (diff_nc_op.f90:19-70 for x = x(j), y = y(k))
        float pj = cx, pl = 0.f, pjk = 0.f, pkl = 0.f, qk = cy, ql = 0.f, qjk = 0.f, qjl = 0.f;
        if constexpr (TER) {
            const float e0 = z1[0] - z0[0], e1 = z1[1] - z0[1], e2 = z1[2] - z0[2], e3 = z1[3] - z0[3];
            const float a = e0 + e1, b = e2 + e3, cx3 = 3.f * cx, cy3 = 3.f * cy;
            const float Zl = a + b, Zj = zm0[0] + zm1[0], Zk = zm0[1] + zm1[1], Zjk = zm0[2] + zm1[2];
            pj = cx3 * Zl;
            pl = cx3 * Zj;
            pjk = cx * (b - a);
            pkl = cx * Zjk;
            qk = cy3 * Zl;
            ql = cy3 * Zk;
            qjk = cy * ((e1 - e0) + (e3 - e2));
            qjl = cy * Zjk;
        }
        // gradient along d of the field with plane sums a below and b above
        auto grad = [&](int d, const M3 (&a)[4], const M3 (&b)[4]) {
            if (d == 2) return cz * (b[0] - a[0]);
            M3 s = d == 0 ? pj * (a[1] + b[1]) : qk * (a[2] + b[2]);
            if (TER) {
                s = m_fma(d == 0 ? pl : ql, b[0] - a[0], s);
                s = m_fma(d == 0 ? pjk : qjk, a[3] + b[3], s);
                s = d == 0 ? m_fma(pkl, b[2] - a[2], s) : m_fma(qjl, b[1] - a[1], s);
            }
            return s;
        };
        M3 G[3];
#pragma unroll
        for (int d = 0; d < 3; d++) G[d] = grad(d, w0, w1);
        if constexpr (PML) {
            // a cell plane below the first node plane is a halo of a
            // partitioned run; the part takes it (its g memory advances here)
            const bool own = owncol && (l >= L0 || l < g.i1node[2]);
#pragma unroll
            for (int d = 0; d < 3; d++) {
                if (!DD[d]) continue;
                long long i, step;
                int p;
                const int sb = mem_of(d, l, false, i, step, p);
                if (sb < 0) continue;
                G[d] = m_fma(A.pmlc[3 * g.npml + p - 1], grad(d, v0, v1), A.pmlc[2 * g.npml + p - 1] * gmem[d]);
                if (own) {
                    float* o = A.gout[sb] + i;
                    o[0] = G[d].x;
                    o[step] = G[d].y;
                    o[2 * step] = G[d].z;
                }
            }
        }
        // strain (the off-diagonal terms twice), stress (2 mu e + lam tr e) / V
        float S[6] = {G[0].x, G[1].y, G[2].z, G[2].y + G[1].z, G[2].x + G[0].z, G[0].y + G[1].x};
        const long long q = g.sz * (long long)(l - 1) + qcol;
        auto inject = [&](const Inject* loc, int nloc, const InjectList& all, float off, float scale) {
            float d[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            apply_inject(loc, nloc, all, q, d, d + 3);
#pragma unroll
            for (int c = 0; c < 3; c++) {
                S[c] = fmaf(d[c], scale, S[c]);
                S[3 + c] = fmaf(off * d[3 + c], scale, S[3 + c]);
            }
        };
        const bool valid = cellcol && l >= g.i1cell[2] && l <= g.i2cell[2];
        const bool src = nsrc && valid && J >= A.ibox[0] && J <= A.ibox[3] && K >= A.ibox[1] && K <= A.ibox[4] &&
                         l >= A.ibox[2] && l <= A.ibox[5];
        if (src && npot != 0) inject(lpot, npot, A.pot, 2.0f, 1.0f);
        {
            const float s = st.x * (S[0] + S[1] + S[2]), m2 = st.y + st.y;
#pragma unroll
            for (int i = 0; i < 3; i++) {
                S[i] = fmaf(m2, S[i], s);
                S[3 + i] = st.y * S[3 + i];
            }
        }
        if (src && nmom != 0) inject(lmom, nmom, A.mom, 1.0f, A.vc[q]);
        if (!PLAIN && A.stats && owncol && (l >= L0 || (PML && l < g.i1node[2])))
            st_w = fmaxn(st_w, (S[0] * S[0] + S[1] * S[1] + S[2] * S[2]) + 2.0f * (S[3] * S[3] + S[4] * S[4] + S[5] * S[5]));
        // modes of the force: divergence of the stress plus the hourglass
        // values yy hourglass_nc (acceleration.f90:22-163)
        const M3 Sx{S[0], S[5], S[4]}, Sy{S[5], S[1], S[3]}, Sz{S[4], S[3], S[2]};
        const float yv = PML ? st.z * A.dh2 : st.z;
        M3 Ejk, Ekl, Ejl, Ejkl, El{}, Ej{}, Ek{};
        // the undamped set: hourglass (interior: whole; shell: viscous)
        if (PML) {
            Ejk = yv * (v0[3] + v1[3]);
            Ekl = yv * (v1[2] - v0[2]);
            Ejl = yv * (v1[1] - v0[1]);
            Ejkl = yv * (v1[3] - v0[3]);
        } else {
            Ejk = yv * (h0[2] + h1[2]);
            Ekl = yv * (h1[1] - h0[1]);
            Ejl = yv * (h1[0] - h0[0]);
            Ejkl = yv * (h1[2] - h0[2]);
        }
        // divergence along the undamped axes
        if (!DD[2]) El = cz * Sz;
        if (!DD[0]) {
            Ej = pj * Sx;
            if (TER) {
                El = DD[2] ? pl * Sx : m_fma(pl, Sx, El);
                Ejk = m_fma(pjk, Sx, Ejk);
                Ekl = m_fma(pkl, Sx, Ekl);
            }
        }
        if (!DD[1]) {
            Ek = qk * Sy;
            if (TER) {
                El = DD[2] && DD[0] ? ql * Sy : m_fma(ql, Sy, El);
                Ejk = m_fma(qjk, Sy, Ejk);
                Ejl = m_fma(qjl, Sy, Ejl);
            }
        }
        m_two<false, hasl>(El, El, acc[0][0], T[0][0]);
        m_two<!(MASK & 1), true>(Ej, Ejl, acc[0][1], T[0][1]);
        m_two<!(MASK & 2), true>(Ek, Ekl, acc[0][2], T[0][2]);
        m_two<true, true>(Ejk, Ejkl, acc[0][3], T[0][3]);
        // divergence along the damped ones
        if constexpr ((MASK & 1) != 0) {
            M3(&a)[4] = acc[SET[0]];
            M3(&t)[4] = T[SET[0]];
            const M3 e = pj * Sx;
            m_two<true, false>(e, e, a[1], t[1]);
            if (TER) {
                const M3 f = pl * Sx, h = pkl * Sx, i = pjk * Sx;
                m_two<false, true>(f, f, a[0], t[0]);
                m_two<false, true>(h, h, a[2], t[2]);
                m_two<true, false>(i, i, a[3], t[3]);
            }
        }
        if constexpr ((MASK & 2) != 0) {
            M3(&a)[4] = acc[SET[1]];
            M3(&t)[4] = T[SET[1]];
            const M3 e = qk * Sy;
            m_two<true, false>(e, e, a[2], t[2]);
            if (TER) {
                const M3 f = ql * Sy, h = qjl * Sy, i = qjk * Sy;
                m_two<false, true>(f, f, a[0], t[0]);
                m_two<false, true>(h, h, a[1], t[1]);
                m_two<true, false>(i, i, a[3], t[3]);
            }
        }
        if constexpr ((MASK & 4) != 0) {
            const M3 e = cz * Sz;
            m_two<false, true>(e, e, acc[SET[2]][0], T[SET[2]][0]);
        }
        if constexpr (PML) {
            // stiffness hourglass
            const float yq = st.z * A.hg1;
            const M3 e = yq * (h1[0] - h0[0]), f = yq * (h1[1] - h0[1]);
            m_two<false, true>(e, e, accq[1], Tq[1]);
            m_two<false, true>(f, f, accq[2], Tq[2]);
            m_two<true, true>(yq * (h0[2] + h1[2]), yq * (h1[2] - h0[2]), accq[3], Tq[3]);
        }
#pragma unroll
        for (int m = 0; m < 4; m++) {
            w0[m] = w1[m];
            if (PML) v0[m] = v1[m];
            if constexpr (TER) z0[m] = z1[m];
        }
#pragma unroll
        for (int m = 0; m < 3; m++) {
            h0[m] = h1[m];
            if constexpr (TER) zm0[m] = zm1[m];
        }
    };

    // ---------------------------------------------------------------- nodes
    // corner values of the force sums of plane l: the thread's own node is
    // corner (1, 1), the other three go to their threads
    M3 own[NSET];
    auto inner = [&](int d, int c) { return !DD[d] || (c >= g.i1pml[d] + 1 && c <= g.i2pml[d] - 1); };
    unsigned in = 0;  // bit c: corner c lies outside the PML along j and k
    if constexpr (PML)
#pragma unroll
        for (int c = 0; c < 4; c++)
            if (inner(0, J + (c & 1)) && inner(1, K + (c >> 1))) in |= 1u << c;
    auto put = [&](int l) {
        float4* X = sX + (L::NB == 2 ? (l & 1) : 0) * (NSET * 3 * NT) + tid;
        const bool inl = PML && inner(2, l);
#pragma unroll
        for (int s = 0; s < NSET; s++) {
            M3 f[4];
            if (s == 0) m_corners<hasl ? 15 : 14>(T[0], f);
            else if (DD[0] && s == SET[0]) m_corners<TER ? 15 : 2>(T[s], f);
            else if (DD[1] && s == SET[1]) m_corners<TER ? 15 : 4>(T[s], f);
            else m_corners<1>(T[s], f);
            if (PML && s == 0) {
                M3 q[4];
                m_corners<14>(Tq, q);
#pragma unroll
                for (int c = 0; c < 4; c++) f[c] = m_fma(inl && (in >> c & 1) ? 1.f : 0.f, q[c], f[c]);
            }
            own[s] = f[3];
#pragma unroll
            for (int c = 0; c < 3; c++)
                X[(3 * s + c) * NT] = make_float4(f[c].x, f[c].y, f[c].z, 0.f);
        }
    };
    auto finish = [&](int l, int slot, float mr) {
        if (!outcol) return;
        const float4* X = sX + (L::NB == 2 ? (l & 1) : 0) * (NSET * 3 * NT) + tid;
        auto get = [&](int i) {
            const float4 a = X[i];
            return M3{a.x, a.y, a.z};
        };
        // corner (0, 0) of the cell past both, (1, 0) of the one a row on, (0, 1) of the next along j
        M3 f[NSET];
#pragma unroll
        for (int s = 0; s < NSET; s++)
            f[s] = (own[s] + get((3 * s + 2) * NT + 1)) + (get((3 * s + 1) * NT + TJ) + get(3 * s * NT + TJ + 1));
        if constexpr (PML) {
            // p memory of the damped axes (acceleration.f90:37-104); the
            // sums are minus the force
#pragma unroll
            for (int d = 0; d < 3; d++) {
                if (!DD[d]) continue;
                M3 s = f[SET[d]];
                long long i, step;
                int p;
                const int sb = mem_of(d, l, true, i, step, p);
                if (sb >= 0) {
                    s = m_fma(A.pmlc[g.npml + p - 1], s, -A.pmlc[p - 1] * pmem[d]);
                    const M3 next = m_fma(-g.dt, s, pmem[d]);
                    float* o = A.sl.p[sb] + i;
                    o[0] = next.x;
                    o[step] = next.y;
                    o[2 * step] = next.z;
                }
                f[0] = f[0] + s;
            }
        }
        const float4* pn = sN + slot * (2 * NP) + (tx + 1) + NJ * (ty + 1);
        const float4 a = pn[0], b = pn[NP];
        const M3 u{a.x, a.y, a.z}, v{b.x, b.y, b.z};
        const long long q = g.sz * (long long)(l - 1) + qnod;
        if ((nsrc && nfrc != 0) || (!PLAIN && (A.fax >= 0 || A.stats))) {
            float fs[3] = {-f[0].x, -f[0].y, -f[0].z};
            const float uv[6] = {u.x, u.y, u.z, v.x, v.y, v.z};
            const Inject* E = nfrc >= 0 ? lfrc : A.force.e;
            const int n = nfrc >= 0 ? nfrc : A.force.n;
            for (int e = 0; e < n; e++)
                if (E[e].idx == q) {
                    const int c = E[e].comp;
                    const float inc = E[e].inc;
                    if (c == 0) fs[0] = fs[0] + inc;
                    else if (c == 1) fs[1] = fs[1] + inc;
                    else fs[2] = fs[2] + inc;
                }
            finish_node<true>(A, q, jn, kn, l, fs, mr, uv, g.dt, st_a, st_v, st_u);
            return;
        }
        const M3 ac = -mr * f[0];
        if (!PLAIN && A.aout[0]) {
            A.aout[0][q] = ac.x;
            A.aout[1][q] = ac.y;
            A.aout[2][q] = ac.z;
        }
        if (PLAIN || A.fold) {
            const float dt = g.dt;
            const M3 vn = m_fma(dt, ac, v), un = m_fma(dt, vn, u);
            A.vout[0][q] = vn.x;
            A.vout[1][q] = vn.y;
            A.vout[2][q] = vn.z;
            A.uout[0][q] = un.x;
            A.uout[1][q] = un.y;
            A.uout[2][q] = un.z;
        }
    };

    // ---------------------------------------------------------------- stream
    // planes L0 - 1 .. L0 + 2 first, one copy group each; then plane l + 4
    // into the slot of plane l - 1 once every thread is done with node
    // plane l - 1, so that two planes are on their way
    int slot = 0;  // of plane l
    auto next_slot = [&](int s, int n) { return s + n >= L::NS ? s + n - L::NS : s + n; };
#pragma unroll 1
    for (int p = -1; p <= 2; p++) {
        fetch(L0 + p, p + 1);
        cp_async_commit();
    }
    float4 nxt = stat_load(L0 - 1);
    cp_async_wait<2>();
    __syncthreads();
    gather(0, plane_damped(L0 - 1), w0, h0, v0, z0, zm0);
#pragma unroll 1
    for (int l = L0 - 1; l <= L1; l++) {
        const float4 cur = nxt;
        nxt = stat_load(l + 1);
#pragma unroll
        for (int d = 0; d < 3; d++) {
            if (!DD[d]) continue;
            gmem[d] = mem_get(d, l, false);
            pmem[d] = mem_get(d, l, true);
        }
        // the sums of plane l were taken for cell plane l - 1
        if (DD[2] && l >= L0 && plane_damped(l) != plane_damped(l - 1))
            gather(slot, plane_damped(l), w0, h0, v0, z0, zm0);
        gather(next_slot(slot, 1), plane_damped(l), w1, h1, v1, z1, zm1);
        cell(l, cur);
        if (l >= L0) put(l);
        cp_async_wait<1>();
        __syncthreads();  // force values of plane l in place, plane l + 2 landed, node plane l - 1 done
        fetch(l + 4, next_slot(slot, 4));
        cp_async_commit();
        if (l >= L0) finish(l, slot, cur.w);
        slot = next_slot(slot, 1);
        if (L::NB == 1) __syncthreads();  // the force values are read
    }
    cp_async_wait_all();
    if (!PLAIN && A.stats) {
        bmax(A.red + 0, st_a);
        bmax(A.red + 1, st_v);
        bmax(A.red + 2, st_u);
        bmax(A.red + 3, st_w);
    }
}
