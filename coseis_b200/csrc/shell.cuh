// PML-shell step kernel in reference order (included by fused.cu): the whole
// step on the node boxes of the PML shell, every operation of the reference
// in its order (see k_interior), with the PML terms of the axes in MASK (bit
// d: axis d may be damped somewhere in the box).
//
// The node ring holds the raw (u, gam), (v, coordinate) of each node as
// 128-bit groups, copied in by cp.async: a cell forms w and the hourglass
// input of its corners from them and, in the PML, differentiates u and v
// themselves.  Cell planes have k_interior's layout (WRITE_CELL), two of
// them.  A PML cell carries the viscous hourglass values in its hourglass
// slots; the layer that is also elastic (next to the inner region) carries
// the elastic ones, and PML nodes form its viscous values from the ring.
//
// One instantiation per class of damped axes: the region tests of the other
// axes are compiled out, a single damped axis has its memories read at the
// start of a plane's work, and the corners come from shared memory, where
// one kernel for all classes took 164 warp instructions per node with 48
// loads per PML cell from device memory.  256 x 256 x 128 terrain, 12-node
// PML: 15.1 -> 12.5 ms for ten steps; the classes also run side by side.  At
// two blocks per SM the classes of one axis spill 150 to 290 bytes a thread.
#pragma once

template <int GEOM>
struct LaySh {
    static constexpr int TJ = SJ, TK = SK, NJ = TJ + 1;
    static constexpr int NP = NJ * (TK + 1), NT = TJ * TK;
    static constexpr int NG = GEOM == GEOM_GENERAL ? 3 : 2;  // (u, gam) (v, coordinate 0) [(coordinates 1, 2)]
    static constexpr int NS = 4;                             // ring slots
    static constexpr int NGC = Lay<GEOM>::NGC, NDIR = Lay<GEOM>::NDIR;
    static constexpr size_t bytes = 16 * (size_t)(NS * NG * NP + 2 * NGC * NT);
};

template <int GEOM, int MASK>
__global__ void __launch_bounds__(SJ * SK, GEOM == GEOM_GENERAL || MASK == 7 ? 1 : 2) k_shell(StepArgs A) {
    using L = LaySh<GEOM>;
    constexpr int TJ = L::TJ, TK = L::TK, NJ = L::NJ, NP = L::NP, NT = L::NT, NG = L::NG, NGC = L::NGC, NDIR = L::NDIR;
    constexpr bool TER = GEOM == GEOM_TERRAIN, GEN = GEOM == GEOM_GENERAL;
    constexpr bool DD[3] = {(MASK & 1) != 0, (MASK & 2) != 0, (MASK & 4) != 0};
    extern __shared__ float4 sm4[];
    float4* sN = sm4;                     // [NS][NG][NP] nodes
    float4* sC = sN + L::NS * NG * NP;    // [2][NGC][NT] cells
    const Geom& g = A.g;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + TJ * ty;
    const int* it = A.items + 6 * blockIdx.x;
    const int j0 = it[0], k0 = it[1], jm = it[2], km = it[3], L0 = it[4], L1 = it[5];
    const int J = j0 - 1 + tx, K = k0 - 1 + ty;  // this thread's cell column
    const int jn = j0 + tx, kn = k0 + ty;        // this thread's node column
    const bool outcol = tx < TJ - 1 && ty < TK - 1 && jn <= jm && kn <= km;
    const bool cellcol = J >= g.i1cell[0] && J <= g.i2cell[0] && K >= g.i1cell[1] && K <= g.i2cell[1];
    const bool owncol = J >= j0 && J <= jm && K >= k0 && K <= km;
    const float h = g.h, dt = g.dt;
    float st_a = 0.f, st_v = 0.f, st_u = 0.f, st_w = 0.f;
    float txa = 0.f, txb = 0.f, tya = 0.f, tyb = 0.f;
    if (TER && cellcol) {
        txa = A.x1d[J - 1];
        txb = A.x1d[J];
        tya = A.y1d[K - 1];
        tyb = A.y1d[K];
    }
    // point sources (see k_interior)
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
    const bool scol = (npot != 0 || nmom != 0) && J >= A.ibox[0] && J <= A.ibox[3] && K >= A.ibox[1] && K <= A.ibox[4];

    // ---------------------------------------------------------------- loads
    // past the mesh the last node or plane is copied: only cells off the
    // mesh and cells that feed no output read it
    constexpr int NR = (NP + NT - 1) / NT;
    unsigned goff[NR];
#pragma unroll
    for (int r = 0; r < NR; r++) {
        const int n = tid + r * NT;
        const int j = min(j0 - 1 + n % NJ, g.nm[0]), k = min(k0 - 1 + n / NJ, g.nm[1]);
        goff[r] = (unsigned)(j - 1) + (unsigned)g.sy * (unsigned)(k - 1);
    }
    auto fetch = [&](int l) {
        if (l > L1 + 1) return;
        const long long pl = g.sz * (long long)(min(max(l, 1), g.nm[2]) - 1);
#pragma unroll
        for (int r = 0; r < NR; r++) {
            if ((r + 1) * NT > NP && tid + r * NT >= NP) continue;
            float* d = reinterpret_cast<float*>(sN + (l & 3) * (NG * NP) + tid + r * NT);
            const long long q = pl + goff[r];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                cp_async4(d + c, A.uin[c] + q);
                cp_async4(d + 4 * NP + c, A.vin[c] + q);
            }
            cp_async4(d + 3, A.gam + q);
            if (TER) cp_async4(d + 4 * NP + 3, A.x[2] + q);
            if (GEN) {
                cp_async4(d + 4 * NP + 3, A.x[0] + q);
                cp_async4(d + 8 * NP, A.x[1] + q);
                cp_async4(d + 8 * NP + 1, A.x[2] + q);
            }
        }
        cp_async_commit();
    };
    float cur[5];  // lam, mu, 1/V, yy of the cell, mr of the node
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
    // PML slab of cell or node c along axis d: near (d) or far (3 + d), its
    // layer and the 1-based damping index.  A cell or node of both (the
    // bands of opposite faces meet) has the far one applied after the near.
    auto near_of = [&](int d, int c, bool node, int& layer, int& p) {
        layer = c - (node ? g.i1node[d] : g.i1cell[d]);
        p = c + g.nnoff[d];
        return DD[d] && c <= g.i1pml[d];
    };
    auto far_of = [&](int d, int c, bool node, int& layer, int& p) {
        layer = (node ? g.i2node[d] : g.i2cell[d]) - c;
        p = g.nn[d] - c - g.nnoff[d] + (node ? 1 : 0);
        return DD[d] && c >= g.i2pml[d] - (node ? 0 : 1);
    };
    // memories of one damped axis, read at the start of a plane's work
    constexpr bool ONE = MASK == 1 || MASK == 2 || MASK == 4;
    constexpr int PD = MASK == 1 ? 0 : MASK == 2 ? 1 : 2;
    float gpre[3] = {0.f, 0.f, 0.f}, ppre[3] = {0.f, 0.f, 0.f};
    auto mem_load = [&](int l) {
        if constexpr (ONE) {
            int layer, p;
            if (cellcol && l >= g.i1cell[2] && l <= g.i2cell[2]) {
                const int c = PD == 0 ? J : PD == 1 ? K : l;
                const int sb = near_of(PD, c, false, layer, p) ? PD : far_of(PD, c, false, layer, p) ? 3 + PD : -1;
                if (sb >= 0)
#pragma unroll
                    for (int ic = 0; ic < 3; ic++) gpre[ic] = A.sl.g[sb][slab_idx(g, PD, A.sl.tg[sb], layer, J, K, l, ic)];
            }
            if (outcol && l >= L0) {
                const int c = PD == 0 ? jn : PD == 1 ? kn : l;
                const int sb = near_of(PD, c, true, layer, p) ? PD : far_of(PD, c, true, layer, p) ? 3 + PD : -1;
                if (sb >= 0)
#pragma unroll
                    for (int ic = 0; ic < 3; ic++) ppre[ic] = A.sl.p[sb][slab_idx(g, PD, A.sl.tp[sb], layer, jn, kn, l, ic)];
            }
        }
    };

    // ---------------------------------------------------------------- cell phase
    auto cells = [&](int l) {
        float4* cw = sC + (l & 1) * (NGC * NT) + tid;
        if (!(cellcol && l >= g.i1cell[2] && l <= g.i2cell[2])) {
#pragma unroll
            for (int i = 0; i < NGC; i++) cw[i * NT] = make_float4(0.f, 0.f, 0.f, 0.f);
            return;
        }
        const long long q = g.idx(J, K, l);
        const int cc[3] = {J, K, l};
        // region of the cell (stress.f90:141-248, acceleration.f90:136-183)
        bool nearS[3], farS[3], anyS = false, inE = true;
        int lay1[3], lay2[3], p1[3], p2[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            nearS[d] = near_of(d, cc[d], false, lay1[d], p1[d]);
            farS[d] = far_of(d, cc[d], false, lay2[d], p2[d]);
            anyS = anyS || nearS[d] || farS[d];
            inE = inE && (!DD[d] || (cc[d] >= g.i1pml[d] && cc[d] <= g.i2pml[d] - 1));
        }
        // a cell plane below the first node plane is a halo of a partitioned run;
        // the part takes it (the PML g memory of that halo cell advances here)
        const bool own = owncol && (l >= L0 || l < g.i1node[2]);
        // corners by corner id n = dj + 2 dk + 4 dl
        float U[3][8], V[3][8], G8[8], X0[8], X1[8], X2[8];
        {
            const float4* q0 = sN + (l & 3) * (NG * NP) + (tx + NJ * ty);
            const float4* q1 = sN + ((l + 1) & 3) * (NG * NP) + (tx + NJ * ty);
#pragma unroll
            for (int n = 0; n < 8; n++) {
                const float4* p = ((n >> 2) ? q1 : q0) + (n & 1) + NJ * ((n >> 1) & 1);
                const float4 a = p[0], b = p[NP];
                U[0][n] = a.x; U[1][n] = a.y; U[2][n] = a.z; G8[n] = a.w;
                V[0][n] = b.x; V[1][n] = b.y; V[2][n] = b.z;
                if (TER) {
                    X0[n] = (n & 1) ? txb : txa;
                    X1[n] = ((n >> 1) & 1) ? tyb : tya;
                    X2[n] = b.w;
                } else if (GEN) {
                    const float2 c = reinterpret_cast<const float2*>(p + 2 * NP)[0];
                    X0[n] = b.w;
                    X1[n] = c.x;
                    X2[n] = c.y;
                }
            }
        }
        float B[3][8];
        float cnb[NDIR > 0 ? NDIR : 1][8];
        if (GEOM == GEOM_RECT) {
#pragma unroll
            for (int a = 0; a < 3; a++)
#pragma unroll
                for (int t = 0; t < 8; t++) B[a][t] = A.br.bnc[a][t];
        } else {
            brackets_nc_g<float>(X1, X2, B[0]);
            cell_cn_brackets_g<float>(X1, X2, B[0], cnb[0], 0.0f);
            brackets_nc_g<float>(X2, X0, B[1]);
            cell_cn_brackets_g<float>(X2, X0, B[1], cnb[NDIR > 1 ? 1 : 0], 0.0f);
            if (TER) {
#pragma unroll
                for (int t = 0; t < 8; t++) B[2][t] = A.br.bnc[2][t];
            } else {
                brackets_nc_g<float>(X0, X1, B[2]);
                cell_cn_brackets_g<float>(X0, X1, B[2], cnb[NDIR > 0 ? NDIR - 1 : 0], 0.0f);
            }
        }
        const bool elastic = A.hourglass && inE, viscous = A.hourglass && A.hgvisc && anyS && !inE;
        float ed[3] = {0.f, 0.f, 0.f}, eo[3] = {0.f, 0.f, 0.f}, he[12];
#pragma unroll
        for (int i = 0; i < 12; i++) he[i] = 0.f;
#pragma unroll
        for (int ic = 0; ic < 3; ic++) {
            // PML cells differentiate u, the others w1 = u + gam * v
            // (time_integration.f90:36)
            float W[8], Vt[8];
#pragma unroll
            for (int t = 0; t < 8; t++) {
                const int n = term_corner(t);
                Vt[t] = V[ic][n];
                W[t] = anyS ? U[ic][n] : U[ic][n] + G8[n] * V[ic][n];
            }
#pragma unroll
            for (int iid = 0; iid < 3; iid++) {
                const int id = (ic + iid + 1) % 3;
                float s;
                if (DD[id] && (nearS[id] || farS[id])) {
                    const float raw = stencil8(Vt, B[id], h);
                    s = raw;
                    if (nearS[id]) {
                        const long long gi = slab_idx(g, id, A.sl.tg[id], lay1[id], J, K, l, ic);
                        const float gm = ONE ? gpre[ic] : A.sl.g[id][gi];
                        s = A.pmlc[3 * g.npml + p1[id] - 1] * raw + A.pmlc[2 * g.npml + p1[id] - 1] * gm;
                        if (own) A.gout[id][gi] = s;
                    }
                    if (farS[id]) {
                        const long long gi = slab_idx(g, id, A.sl.tg[3 + id], lay2[id], J, K, l, ic);
                        const float gm = ONE && !nearS[id] ? gpre[ic] : A.sl.g[3 + id][gi];
                        s = A.pmlc[3 * g.npml + p2[id] - 1] * raw + A.pmlc[2 * g.npml + p2[id] - 1] * gm;
                        if (own) A.gout[3 + id][gi] = s;
                    }
                } else {
                    s = stencil8(W, B[id], h);
                }
                if (ic == id) ed[ic] = s;
                else if (ic < id) eo[3 - ic - id] = 0.5f * s;
                else eo[3 - ic - id] = eo[3 - ic - id] + 0.5f * s;
            }
            // hourglass cell values: elastic, yy hourglass_nc(hg1 u + dt hg2 v),
            // or on PML cells away from the elastic region viscous,
            // dt hg2 yy hourglass_nc(v) (acceleration.f90:141-183)
            if (elastic || viscous) {
                const float y = elastic ? cur[3] : A.dh2 * cur[3];
                float H[8];
#pragma unroll
                for (int t = 0; t < 8; t++) {
                    const int n = hg_corner(t);
                    H[t] = elastic ? A.hg1 * U[ic][n] + A.dh2 * V[ic][n] : V[ic][n];
                }
#pragma unroll
                for (int iq = 0; iq < 4; iq++) he[3 * iq + ic] = hg_sum(H, iq) * y;
            }
        }
        const bool src = scol && l >= A.ibox[2] && l <= A.ibox[5];
        if (src) apply_inject(lpot, npot, A.pot, q, ed, eo);
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
        if (A.stats && own)
            st_w = fmaxn(st_w, (ed[0] * ed[0] + ed[1] * ed[1] + ed[2] * ed[2]) + 2.0f * (eo[0] * eo[0] + eo[1] * eo[1] + eo[2] * eo[2]));
        cw[0] = make_float4(ed[0], ed[1], ed[2], eo[0]);
        cw[NT] = make_float4(eo[1], eo[2], he[0], he[1]);
        cw[2 * NT] = make_float4(he[3], he[4], he[6], he[7]);
        cw[3 * NT] = make_float4(he[9], he[10], he[2], he[5]);
        cw[4 * NT] = make_float4(he[8], he[11], 0.f, 0.f);
        if constexpr (NDIR >= 2) {
#pragma unroll
            for (int q2 = 0; q2 < 4; q2++)
                cw[(5 + q2) * NT] = make_float4(cnb[0][2 * q2], cnb[1][2 * q2], cnb[0][2 * q2 + 1], cnb[1][2 * q2 + 1]);
        }
        if constexpr (NDIR == 3) {
            cw[9 * NT] = make_float4(cnb[2][0], cnb[2][1], cnb[2][2], cnb[2][3]);
            cw[10 * NT] = make_float4(cnb[2][4], cnb[2][5], cnb[2][6], cnb[2][7]);
        }
    };

    // ---------------------------------------------------------------- node phase
    auto nodes = [&](int l) {
        if (!outcol) return;
        const long long q = g.idx(jn, kn, l);
        const float4* c0 = sC + ((l - 1) & 1) * (NGC * NT) + tid;  // cell plane l-1
        const float4* c1 = sC + (l & 1) * (NGC * NT) + tid;        // cell plane l
        auto cpos = [&](int p) { return ((p >> 2) ? c1 : c0) + (p & 1) + TJ * ((p >> 1) & 1); };
        auto pt = [](int t) { return (t & 1) + 2 * (t >> 2) + 4 * ((t >> 1) & 1); };
        auto ph = [](int t) {
            const int o = hg_corner(t);
            return (1 - (o & 1)) + 2 * (1 - ((o >> 1) & 1)) + 4 * (1 - (o >> 2));
        };
        float S[6][8], Bc[3][8];
#pragma unroll
        for (int t = 0; t < 8; t++) {
            const float4* cp = cpos(pt(t));
            const float4 a = cp[0];
            const float2 b = reinterpret_cast<const float2*>(cp + NT)[0];
            S[0][t] = a.x; S[1][t] = a.y; S[2][t] = a.z; S[3][t] = a.w; S[4][t] = b.x; S[5][t] = b.y;
            if (NDIR >= 2) {
                const float2 bb = reinterpret_cast<const float2*>(cp + (5 + t / 2) * NT)[t % 2];
                Bc[0][t] = bb.x;
                Bc[1][t] = bb.y;
            }
            if (NDIR == 3) Bc[2][t] = reinterpret_cast<const float*>(cp + (9 + t / 4) * NT)[t % 4];
            if (GEOM == GEOM_RECT)
#pragma unroll
                for (int id = 0; id < 3; id++) Bc[id][t] = A.br.bcn[id][t];
            if (TER) Bc[2][t] = A.br.bcn[2][t];
        }
        float f[3];
#pragma unroll
        for (int ic = 0; ic < 3; ic++) {
#pragma unroll
            for (int iid = 0; iid < 3; iid++) {
                const int id = (ic + iid) % 3;
                const int comp = ic == id ? ic : 3 + (3 - ic - id);
                float s = stencil8(S[comp], Bc[id], h);
                if (DD[id]) {
                    const int c = id == 0 ? jn : id == 1 ? kn : l;
                    int layer, p;
                    const bool nr = near_of(id, c, true, layer, p);
                    if (nr) {
                        float* P = A.sl.p[id] + slab_idx(g, id, A.sl.tp[id], layer, jn, kn, l, ic);
                        const float m = ONE ? ppre[ic] : *P;
                        s = A.pmlc[g.npml + p - 1] * s + A.pmlc[p - 1] * m;
                        *P = m + dt * s;
                    }
                    if (far_of(id, c, true, layer, p)) {
                        float* P = A.sl.p[3 + id] + slab_idx(g, id, A.sl.tp[3 + id], layer, jn, kn, l, ic);
                        const float m = ONE && !nr ? ppre[ic] : *P;
                        s = A.pmlc[g.npml + p - 1] * s + A.pmlc[p - 1] * m;
                        *P = m + dt * s;
                    }
                }
                f[ic] = iid == 0 ? s : f[ic] + s;
            }
        }
        if (A.hourglass) {
            const int cn_[3] = {jn, kn, l};
            bool ne = true;
#pragma unroll
            for (int d = 0; d < 3; d++) ne = ne && (!DD[d] || (cn_[d] >= g.i1pml[d] + 1 && cn_[d] <= g.i2pml[d] - 1));
            if (ne || A.hgvisc) {
                // each cell's hourglass groups by hourglass_cn term; a PML
                // node takes the viscous values of the elastic layer's cells
                // from v, and zero from cells outside the mesh
                float H[4][3][8];
#pragma unroll
                for (int t = 0; t < 8; t++) {
                    const float4* cp = cpos(ph(t));
                    const float2 g1 = reinterpret_cast<const float2*>(cp + NT)[1];
                    const float4 g2 = cp[2 * NT], g3 = cp[3 * NT];
                    const float2 g4 = reinterpret_cast<const float2*>(cp + 4 * NT)[0];
                    H[0][0][t] = g1.x; H[0][1][t] = g1.y; H[0][2][t] = g3.z;
                    H[1][0][t] = g2.x; H[1][1][t] = g2.y; H[1][2][t] = g3.w;
                    H[2][0][t] = g2.z; H[2][1][t] = g2.w; H[2][2][t] = g4.x;
                    H[3][0][t] = g3.x; H[3][1][t] = g3.y; H[3][2][t] = g4.y;
                }
                if (!ne) {
#pragma unroll
                    for (int t = 0; t < 8; t++) {
                        const int o = hg_corner(t);
                        const int Jc = jn - (o & 1), Kc = kn - ((o >> 1) & 1), Lc = l - (o >> 2);
                        const int cc[3] = {Jc, Kc, Lc};
                        bool real = true, inEc = true;
#pragma unroll
                        for (int d = 0; d < 3; d++) {
                            real = real && cc[d] >= g.i1cell[d] && cc[d] <= g.i2cell[d];
                            inEc = inEc && (!DD[d] || (cc[d] >= g.i1pml[d] && cc[d] <= g.i2pml[d] - 1));
                        }
                        if (!(real && inEc)) continue;
                        // the cell's corners in the ring: plane slots Lc, Lc + 1
                        const float yc = A.dh2 * A.yy[g.idx(Jc, Kc, Lc)];
                        const int n0 = (Jc - (j0 - 1)) + NJ * (Kc - (k0 - 1));
                        float4 Vc[8];
#pragma unroll
                        for (int m = 0; m < 8; m++) {
                            const int n = hg_corner(m);
                            Vc[m] = sN[((Lc + (n >> 2)) & 3) * (NG * NP) + NP + n0 + (n & 1) + NJ * ((n >> 1) & 1)];
                        }
#pragma unroll
                        for (int ic = 0; ic < 3; ic++) {
                            float v8[8];
#pragma unroll
                            for (int m = 0; m < 8; m++) v8[m] = ic == 0 ? Vc[m].x : ic == 1 ? Vc[m].y : Vc[m].z;
#pragma unroll
                            for (int iq = 0; iq < 4; iq++) H[iq][ic][t] = yc * hg_sum(v8, iq);
                        }
                    }
                }
#pragma unroll
                for (int iq = 0; iq < 4; iq++)
#pragma unroll
                    for (int ic = 0; ic < 3; ic++) f[ic] = f[ic] - hg_sum(H[iq][ic], iq);
            }
        }
        if (nfrc != 0) {
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
        }
        const float4* pn = sN + (l & 3) * (NG * NP) + (tx + 1) + NJ * (ty + 1);
        const float4 a = pn[0], b = pn[NP];
        const float uv[6] = {a.x, a.y, a.z, b.x, b.y, b.z};
        finish_node<false>(A, q, jn, kn, l, f, cur[4], uv, dt, st_a, st_v, st_u);
    };

    // ---------------------------------------------------------------- stream
    // ring: planes L0 - 1 .. L0 + 1, then plane l + 3 into the slot of plane
    // l - 1 once node plane l is done with it
#pragma unroll 1
    for (int p = -1; p <= 1; p++) fetch(L0 + p);
    stat_load(L0 - 1, cur);
    cp_async_wait_all();
    __syncthreads();
    fetch(L0 + 2);
    // (one call of each phase, so that both are inlined)
#pragma unroll 1
    for (int l = L0 - 1; l <= L1; l++) {
        mem_load(l);
        cells(l);
        float nxt[5];
        stat_load(l + 1, nxt);
        if (l >= L0) {
            cp_async_wait_all();
            __syncthreads();  // cell plane l complete, plane l + 2 landed
            nodes(l);
            __syncthreads();  // cell plane l - 1 and ring slot l - 1 free
            fetch(l + 3);
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
}
