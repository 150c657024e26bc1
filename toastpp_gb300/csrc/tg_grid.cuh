// tg_grid.cuh -- the grid-basis Jacobian of a pixel raster.
//
// Reference: GenerateJacobian_grid (src/libstoast/jacobian.cc:289-373,
// complex, projections given) and GenerateJacobian_cw_grid (516-712, real)
// with Raster_Pixel (raster_px.cc:10-48).  The PMDFs are formed on the
// raster's grid; where the basis is coarser than the grid (an intermediate
// grid) the rows are then mapped to the basis by G (grid_to_sol_rows_kernel).
//
// Per request the fields (source-major, natural numbering) are resampled on
// the grid column by column (gm[c * glen + g]), then the values and the
// central or one-sided differences of ImageGradient (jacobian.cc:944-1060) at
// the solution points (the grid points inside the mesh) go to planes
// P[(c * (1 + dim) + comp) * slen + s] (comp 0 the value, 1..dim the
// gradient), so that a thread per solution point reads every plane of a
// source or detector coalesced.  Then one thread per solution point and
// group of sources walks the sources' links and writes its column of every
// link row.
#pragma once
#include "tg_jac.cuh"

namespace tg {

struct GridDev {
    int dim, nx, ny, nz, glen, slen;
    double ih[3];                // 1 / (gsize / n) per axis (ImageGradient's spacing)
    const int* elref;            // glen: containing element or -1
    const int* sol;              // slen: grid index of each solution point
    const int* rowptr;           // glen + 1: grid map matrix B (natural node columns)
    const int* col;
    const double* val;
};

// Map_MeshToGrid (raster.cc:188-199; complex: Ax_cplx, crmatrix_imp.hpp:
// 1302-1327): gm[g * k + c] = sum_j B(g, j) x[row(col_j) * ld + c], x
// node-major, rows in the natural numbering (perm null) or in a layout
// (row = perm[natural]); a warp per grid point, lanes over columns
template <class V>
__global__ void grid_map_kernel(GridDev G, int k, const V* __restrict__ x, int ld, const int* __restrict__ perm,
                                V* __restrict__ gm)
{
    const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (g >= G.glen) return;
    const int j0 = G.rowptr[g], j1 = G.rowptr[g + 1];
    for (int c = lane; c < k; c += 32) {
        V acc = vzero<V>();
        for (int j = j0; j < j1; j++) {
            const int r = perm ? perm[G.col[j]] : G.col[j];
            acc = vadd(acc, vscale(x[(size_t)r * ld + c], G.val[j]));
        }
        gm[(size_t)g * k + c] = acc;
    }
}

// value (comp 0) or ImageGradient component comp - 1 of column c at grid
// point g: central or one-sided differences as jacobian.cc:944-1060 takes
// them; masked: neighbours outside the element mask do not count, else every
// grid point does
template <class V>
__device__ __forceinline__ V grid_component(const GridDev& G, int k, const V* __restrict__ gm, int g, int c,
                                            int comp, int masked)
{
    const V v0 = gm[(size_t)g * k + c];
    if (comp == 0) return v0;
    const int d = comp - 1;
    const int co = d == 0 ? g % G.nx : (d == 1 ? (g / G.nx) % G.ny : g / (G.nx * G.ny));
    const int len = d == 0 ? G.nx : (d == 1 ? G.ny : G.nz), st = d == 0 ? 1 : (d == 1 ? G.nx : G.nx * G.ny);
    const bool blo = co > 0 && (!masked || G.elref[g - st] >= 0);
    const bool bhi = co < len - 1 && (!masked || G.elref[g + st] >= 0);
    using R = typename vt<V>::R;
    if (blo && bhi) return vscale(vsub(gm[(size_t)(g + st) * k + c], gm[(size_t)(g - st) * k + c]), (R)(0.5 * G.ih[d]));
    // a point outside the mask (a blob basis's solution point off the
    // mesh) without both neighbours inside: 0 (ImageGradient,
    // jacobian.cc:944-1060)
    if (masked && G.elref[g] < 0) return vzero<V>();
    if (blo) return vscale(vsub(v0, gm[(size_t)(g - st) * k + c]), (R)G.ih[d]);
    if (bhi) return vscale(vsub(gm[(size_t)(g + st) * k + c], v0), (R)G.ih[d]);
    return vzero<V>();
}

// Field planes P[(c * (1 + dim) + comp) * slen + s] from the grid fields:
// block = 32 solution points x 32 columns; each component is formed with
// lanes over columns (coalesced reads of gm) into a shared tile, then
// written with lanes over solution points (coalesced planes)
template <class V, class OUT>
__global__ void __launch_bounds__(256) grid_planes_kernel(GridDev G, int k, const V* __restrict__ gm, int masked,
                                                          OUT* __restrict__ planes)
{
    __shared__ OUT tile[32][33];
    const int s0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
    const int np = 1 + G.dim;
    for (int comp = 0; comp < np; comp++) {
        for (int r = ty; r < 32; r += 8) {
            const int s = s0 + r, c = c0 + tx;
            if (s < G.slen && c < k) tile[r][tx] = vcast<OUT, V>(grid_component(G, k, gm, G.sol[s], c, comp, masked));
        }
        __syncthreads();
        for (int r = ty; r < 32; r += 8) {
            const int c = c0 + r, s = s0 + tx;
            if (s < G.slen && c < k) planes[((size_t)c * np + comp) * G.slen + s] = tile[tx][r];
        }
        __syncthreads();
    }
}

// Map_MeshToGrid of source-major columns, column-major result:
// gm[c * glen + g] = sum_j B(g, j) x[c * n + col_j] in the arithmetic type A;
// columns c < k0 from x0, the others from x1.  A thread per grid point keeps
// its row of B (at most four entries for linear elements) in registers for
// MAPC columns; neighbouring grid points gather from neighbouring nodes.
constexpr int MAPC = 8, MAPU = 4;
template <class A, class V>
__global__ void __launch_bounds__(256) grid_map_cm_kernel(GridDev G, int n, int k, int k0, const V* __restrict__ x0,
                                                          const V* __restrict__ x1, A* __restrict__ gm)
{
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= G.glen) return;
    using R = typename vt<A>::R;
    const int j0 = G.rowptr[g], nj = G.rowptr[g + 1] - j0;
    int col[4];
    R w[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        col[j] = j < nj ? G.col[j0 + j] : 0;
        w[j] = j < nj ? (R)G.val[j0 + j] : (R)0;
    }
    const int c0 = blockIdx.y * MAPC, c1 = min(k, c0 + MAPC);
    auto column = [&](int c) { return c < k0 ? x0 + (size_t)c * n : x1 + (size_t)(c - k0) * n; };
    if (nj > 4) {
        for (int c = c0; c < c1; c++) {
            const V* x = column(c);
            A acc = vzero<A>();
            for (int j = j0; j < j0 + nj; j++) acc = vadd(acc, vscale(vcast<A, V>(x[G.col[j]]), (R)G.val[j]));
            gm[(size_t)c * G.glen + g] = acc;
        }
        return;
    }
    // the gathers of MAPU columns are in flight together (a missing entry
    // gathers node 0 and is not added)
    for (int c = c0; c < c1; c += MAPU) {
        V v[MAPU][4];
#pragma unroll
        for (int u = 0; u < MAPU; u++) {
            const V* x = column(min(c + u, c1 - 1));
#pragma unroll
            for (int j = 0; j < 4; j++) v[u][j] = x[col[j]];
        }
#pragma unroll
        for (int u = 0; u < MAPU; u++) {
            A acc = vzero<A>();
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const A t = vadd(acc, vscale(vcast<A, V>(v[u][j]), w[j]));
                acc = j < nj ? t : acc;
            }
            if (c + u < c1) gm[(size_t)(c + u) * G.glen + g] = acc;
        }
    }
}

// Field planes P[(c * (1 + dim) + comp) * slen + s] from the column-major grid
// fields: a thread per solution point finds, once, the neighbours and weight
// of each axis's difference under the masked and the unmasked rule of
// grid_component, then forms MAPC columns; columns c < kmask are masked, the
// others when mask_rest is set.  Reads and writes run along s.
template <class A>
__global__ void __launch_bounds__(256) grid_planes_cm_kernel(GridDev G, int k, int kmask, int mask_rest,
                                                             const A* __restrict__ gm, A* __restrict__ planes)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= G.slen) return;
    using R = typename vt<A>::R;
    const int g = G.sol[s], np = 1 + G.dim;
    const int co[3] = {g % G.nx, (g / G.nx) % G.ny, g / (G.nx * G.ny)};
    const int len[3] = {G.nx, G.ny, G.nz}, st[3] = {1, G.nx, G.nx * G.ny};
    int lo[2][3], hi[2][3];
    R w[2][3];
#pragma unroll
    for (int mk = 0; mk < 2; mk++)
#pragma unroll
        for (int d = 0; d < 3; d++) {
            lo[mk][d] = hi[mk][d] = g;
            w[mk][d] = (R)0;
            if (d >= G.dim) continue;
            const bool blo = co[d] > 0 && (!mk || G.elref[g - st[d]] >= 0);
            const bool bhi = co[d] < len[d] - 1 && (!mk || G.elref[g + st[d]] >= 0);
            // one-sided differences only at points inside the mask
            const bool in = !mk || G.elref[g] >= 0;
            if (blo) lo[mk][d] = g - st[d];
            if (bhi) hi[mk][d] = g + st[d];
            if ((blo && bhi) || (in && (blo || bhi))) w[mk][d] = (R)((blo && bhi ? 0.5 : 1.0) * G.ih[d]);
        }
    const int c0 = blockIdx.y * MAPC, c1 = min(k, c0 + MAPC);
    for (int c = c0; c < c1; c += MAPU) {
        A v[MAPU], vl[MAPU][3], vh[MAPU][3];
#pragma unroll
        for (int u = 0; u < MAPU; u++) {
            const int cu = min(c + u, c1 - 1);
            const bool mk = cu < kmask || mask_rest;
            const A* x = gm + (size_t)cu * G.glen;
            v[u] = x[g];
#pragma unroll
            for (int d = 0; d < 3; d++)
                if (d < G.dim) {
                    vl[u][d] = x[mk ? lo[1][d] : lo[0][d]];
                    vh[u][d] = x[mk ? hi[1][d] : hi[0][d]];
                }
        }
#pragma unroll
        for (int u = 0; u < MAPU; u++) {
            if (c + u >= c1) break;
            const bool mk = c + u < kmask || mask_rest;
            A* P = planes + (size_t)(c + u) * np * G.slen + s;
            P[0] = v[u];
#pragma unroll
            for (int d = 0; d < 3; d++)
                if (d < G.dim) P[(size_t)(d + 1) * G.slen] = vscale(vsub(vh[u][d], vl[u][d]), mk ? w[1][d] : w[0][d]);
        }
    }
}

// One launch before the grid and element kernels: the factor of each link's
// row, sc / y for log data (Smith's division for complex y), sc for linear
// data (y null), formed in FP64 and cast to the Jacobian's arithmetic type;
// and with x given the cast of the cnt0 source and cnt1 detector values into
// it, one after the other (three launches of 2-4 us each as separate kernels).
template <class C, class V64>
__global__ void grid_prep_kernel(size_t cnt0, const V64* __restrict__ x0, size_t cnt1, const V64* __restrict__ x1,
                                 C* __restrict__ x, int nqm, const V64* __restrict__ y, double sc,
                                 C* __restrict__ ysc)
{
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i < (size_t)nqm) {
        if constexpr (vt<V64>::cplx) {
            const cd r = y ? cdiv(cd{1.0, 0.0}, y[i]) : cd{1.0, 0.0};
            ysc[i] = vcast<C, cd>(cd{r.x * sc, r.y * sc});
        } else {
            ysc[i] = vcast<C, double>(y ? sc / y[i] : sc);
        }
    }
    if (x && i < cnt0 + cnt1) x[i] = vcast<C, V64>(i < cnt0 ? x0[i] : x1[i - cnt0]);
}

// J stores bypass L2 retention (evict-first), so the 2.4 GB stream of rows
// does not push the field planes out of L2
__device__ __forceinline__ void st_stream(float* p, float v) { __stcs(p, v); }
__device__ __forceinline__ void st_stream(double* p, double v) { __stcs(p, v); }

// The links of a block's GQ sources and at most LT detectors in shared
// memory: which sources link to the detector, the offset of the link's J row
// and its factor, read by every thread of the block from there instead of from
// the pair table and the factor array.
constexpr int LT = 64;
template <class V, int GQ>
struct LinkTile {
    unsigned on[LT];
    long long row[GQ][LT];
    V y[GQ][LT];
    // detectors m0 .. m1 - 1 of sources q0 .. q0 + GQ - 1; rows of cols
    // entries, the first of link l0
    __device__ __forceinline__ void fill(int m0, int m1, int q0, int nq, int nm, const int* __restrict__ pair,
                                         const V* __restrict__ ysc, long long cols, int l0)
    {
        for (int j = threadIdx.x; j < m1 - m0; j += blockDim.x) {
            unsigned b = 0;
            for (int g = 0; g < GQ && q0 + g < nq; g++) {
                const int k = pair[(size_t)(q0 + g) * nm + m0 + j];
                if (k < 0) continue;
                b |= 1u << g;
                row[g][j] = (k - l0) * cols;
                y[g][j] = ysc[k];
            }
            on[j] = b;
        }
        __syncthreads();
    }
};

// Sums of products f h of one link: F a source's value, H a detector's, both in
// the form the sum takes.  Complex FP32 runs on packed pairs: the sums of
// (hr, hr) f and (hi, hi) f, whose difference and sum cross-wise is the product
// (a packed multiply-add is one instruction for two, and these kernels are
// bound by instruction issue).
template <class V>
struct LinkSum {
    using F = V;
    using H = V;
    V a = vzero<V>();
    static __device__ __forceinline__ F src(V f) { return f; }
    static __device__ __forceinline__ H det(V h) { return h; }
    static __device__ __forceinline__ V prod(F f, H h) { return vmul(f, h); }
    static __device__ __forceinline__ F sub(F a, F b) { return vsub(a, b); }
    __device__ __forceinline__ void add(F f, H h) { a = vfma(a, f, h); }
    __device__ __forceinline__ V get() const { return a; }
};
template <>
struct LinkSum<cf> {
    using F = unsigned long long;
    struct H {
        unsigned long long r, i;
    };
    unsigned long long p = 0ull, q = 0ull;
    // one product alone: a rounding fewer, and no more instructions
    static __device__ __forceinline__ cf prod(F f, H h)
    {
        const float2 a = f2_unpack(f);
        return vmul(cf{a.x, a.y}, cf{f2_unpack(h.r).x, f2_unpack(h.i).x});
    }
    static __device__ __forceinline__ F src(cf f) { return f2_pack(f.x, f.y); }
    static __device__ __forceinline__ H det(cf h) { return H{f2_pack(h.x, h.x), f2_pack(h.y, h.y)}; }
    static __device__ __forceinline__ F sub(F a, F b) { return f2_sub(a, b); }
    __device__ __forceinline__ void add(F f, H h)
    {
        p = f2_fma(h.r, f, p);
        q = f2_fma(h.i, f, q);
    }
    __device__ __forceinline__ cf get() const
    {
        const float2 a = f2_unpack(p), b = f2_unpack(q);
        return cf{a.x - b.y, a.y + b.x};
    }
};

// the four (real: two) J entries of a link at column e of rows row and row +
// half: mua in the first, kappa in the second half of the columns
template <class V, class JT>
__device__ __forceinline__ void put_link(JT* __restrict__ j0, long long row, long long half, long long kap, V pm, V pk)
{
    JT* r = j0 + row;
    if constexpr (vt<V>::cplx) {
        st_stream(r, (JT)re(pm));
        st_stream(r + kap, (JT)re(pk));
        st_stream(r + half, (JT)im(pm));
        st_stream(r + half + kap, (JT)im(pk));
    } else {
        st_stream(r, (JT)pm);
        st_stream(r + half, (JT)pk);
    }
}

// One thread per (solution point, group of GQ sources): the sources' planes
// stay in registers while the detectors' planes stream past, each loaded once
// per group, the next detector's while this one's entries form.  PMDF_mua =
// -(f a), PMDF_kap = -sum_d (grad_d f)(grad_d a) (jacobian.cc:58-72); LOG
// data are divided by y (complex: PMDF_log, 76-79; real:
// GenerateJacobian_cw, 178-193) and every entry is multiplied by the voxel
// scale (365-370).  ysc[l] carries -scale / y of the link (-scale for LINEAR
// data), so an entry costs one complex product more than its PMDF: a
// division per entry would run on the FP64 pipe.  NP = 1 + dim planes.
// pair[q * nm + m]: link index or -1.  J rows: complex [Re mua | Re kap] at l
// and [Im mua | Im kap] at nQM + l (2 slen columns); real mua at l and kap at
// nQM + l (slen).  With l0 > 0 the kernel serves the sources of one chunk
// whose links are l0 .. l0 + nqm - 1: row l - l0 and nqm + l - l0.
// blockIdx.z: chunks of mc detectors, at most LT.
// FP32 is bound by the plane loads' latency and the J stream (32^3 points, 80 x
// 80 links, 2.4 GB: 644 -> 578 us a call; this kernel for 40 x 80 252 -> 241 us,
// 5 TB/s of the 7.6 a plain write stream reaches, with 82 -> 56 instructions a
// link; groups of 4 and 256 threads 256 us), FP64 by its pipe (6 complex
// products a link: 6.5 ms, of which they take about 6.2).  8 sources a group for
// FP32: half the plane loads of 4; 4 for FP64, where 8 leaves SMs idle at medium
// sizes (disc 40^2, 15 x 17: 79 -> 98 us a call).  Two points a
// thread on packed pairs halve the instructions but lose (FP32 complex 577 ->
// 967 us: eight store streams a warp).
template <class V, class JT, int GQ, int NP>
__global__ void __launch_bounds__(128) grid_jacobian_kernel(int slen, int nq, int nm, int nqm, const V* __restrict__ Fp,
                                                            const V* __restrict__ Ap, const int* __restrict__ pair,
                                                            const V* __restrict__ ysc, JT* __restrict__ J, int l0,
                                                            int mc)
{
    using LS = LinkSum<V>;
    __shared__ LinkTile<V, GQ> tile;
    const int q0 = blockIdx.y * GQ, m0 = blockIdx.z * mc, m1 = min(m0 + mc, nm);
    constexpr bool CPLX = vt<V>::cplx;
    const long long cols = CPLX ? 2 * (long long)slen : (long long)slen, half = nqm * cols;
    tile.fill(m0, m1, q0, nq, nm, pair, ysc, cols, l0);
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= slen) return;
    typename LS::F f[GQ][NP];
#pragma unroll
    for (int g = 0; g < GQ; g++)
#pragma unroll
        for (int d = 0; d < NP; d++) f[g][d] = LS::src(Fp[((size_t)min(q0 + g, nq - 1) * NP + d) * slen + s]);
    JT* j0 = J + s;
    V an[NP];
    const V* ap = Ap + (size_t)m0 * NP * slen + s;
#pragma unroll
    for (int d = 0; d < NP; d++) an[d] = ap[(size_t)d * slen];
    for (int m = m0; m < m1; m++) {
        const int jt = m - m0;
        const unsigned on = tile.on[jt];
        typename LS::H a[NP];
        ap += (size_t)NP * slen;
#pragma unroll
        for (int d = 0; d < NP; d++) {
            a[d] = LS::det(an[d]);
            if (m + 1 < m1) an[d] = ap[(size_t)d * slen];
        }
        if (!on) continue;
#pragma unroll
        for (int g = 0; g < GQ; g++) {
            if (!(on >> g & 1)) continue;
            LS pk;
            const V pm = LS::prod(f[g][0], a[0]);
#pragma unroll
            for (int d = 1; d < NP; d++) pk.add(f[g][d], a[d]);
            const V y = tile.y[g][jt];
            put_link<V, JT>(j0, tile.row[g][jt], half, slen, vmul(pm, y), vmul(pk.get(), y));
        }
    }
}

// Element-basis Jacobian (GenerateJacobian_mesh with elbasis, jacobian.cc:
// 441-497; CW 738-802 and the LOG scaling 178-193), with IntFG_el /
// IntGradFGradG_el (884-939): per element e and link (q, m),
// sum_ij f_i g_j IntFF(i,j) and sum_ij f_i g_j IntDD(i,j).  With h = IntFF g
// (size (1 + [i = j]) / 12 for triangles, / 20 for tetrahedra) the first is
// sum_i f_i h_i; the rows and columns of IntDD sum to zero, so with the
// differences d_i = f_i - f_0 the second is
// sum_{i,j > 0} d_i IntDD(i,j) (g_j - g_0): no cancellation between its terms
// (FP32, error in L2 against FP64: 61-ring disc 5.4e-7 -> 0.9e-7), and NN - 1
// products.  FP64 keeps the d_i and forms the first sum from them too, f_0
// sum_i h_i + sum_{i > 0} d_i h_i: subtractions per link would cost its pipe a
// sixth.  The detector's side is formed once per (element, detector) and shared
// by the group's GQ sources.
// NN nodes per element (3 or 4).  Fields source-major in the natural
// numbering.  ysc[l] = -1 / y for LOG data, -1 for LINEAR.  J: complex
// (2 nQM) x (2 ne) rows -Re / -Im, kappa at column ne + e; real (2 nQM) x ne
// [mua ; kappa].
// blockIdx.z: chunks of mc detectors, at most LT, from detector mb on.
// FP32 is bound by instruction issue, then by the J stream (38.9k tetrahedra,
// 80 x 80 links, 4 GB: 838 -> 734 us a call, 5.4 TB/s), FP64 by its pipe (21.1
// -> 17.6 ms; 9 complex products a link are 15.4).  8 sources a group: the detector's
// side costs as much as 4 links (groups of 4 / 6 / 8: 960 / 810 / 726 us FP32,
// 20.1 / 18.5 / 17.6 ms FP64).
template <class V, class JT, int GQ, int NN>
__global__ void __launch_bounds__(128) element_jacobian_kernel(MeshDev m, int nq, int nm, int nqm,
                                                               const V* __restrict__ F, const V* __restrict__ A,
                                                               const int* __restrict__ pair,
                                                               const V* __restrict__ ysc, JT* __restrict__ J,
                                                               int mc, int mb)
{
    using LS = LinkSum<V>;
    __shared__ LinkTile<V, GQ> tile;
    const int q0 = blockIdx.y * GQ, m0 = mb + blockIdx.z * mc, m1 = min(m0 + mc, nm);
    constexpr bool CPLX = vt<V>::cplx;
    const long long cols = CPLX ? 2 * (long long)m.ne : (long long)m.ne, half = nqm * cols;
    tile.fill(m0, m1, q0, nq, nm, pair, ysc, cols, 0);
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= m.ne) return;
    using R = typename vt<V>::R;
    const int n = m.n;
    const int* nd = m.el + (size_t)e * NN;
    const double* r = m.rec + (size_t)e * EL_REC;
    constexpr double ff = NN == 3 ? 1.0 / 12.0 : 1.0 / 20.0;
    const R cff = (R)(ff * r[0]), cf0 = (R)(ff * (NN + 1) * r[0]);
    R wdd[NN - 1][NN - 1];
    int node[NN];
#pragma unroll
    for (int i = 0; i < NN; i++) node[i] = nd[i];
#pragma unroll
    for (int i = 1; i < NN; i++)
#pragma unroll
        for (int j = 1; j < NN; j++)
            // IntDD: the record's value for triangles, 4 x it for tetrahedra
            wdd[i - 1][j - 1] = (R)((NN == 4 ? 4.0 : 1.0) * r[1 + i * NN + j]);
    constexpr bool DIFF = sizeof(JT) == 8;
    typename LS::F f[GQ][NN];
#pragma unroll
    for (int g = 0; g < GQ; g++) {
        const V* x = F + (size_t)min(q0 + g, nq - 1) * n;
        const V x0 = x[node[0]];
        f[g][0] = LS::src(x0);
#pragma unroll
        for (int i = 1; i < NN; i++) f[g][i] = LS::src(DIFF ? vsub(x[node[i]], x0) : x[node[i]]);
    }
    JT* j0 = J + e;
    // the next detector's nodal values load while this one's entries form
    V an[NN];
    const V* ap = A + (size_t)m0 * n;
#pragma unroll
    for (int j = 0; j < NN; j++) an[j] = ap[node[j]];
    for (int mm = m0; mm < m1; mm++) {
        const int jt = mm - m0;
        const unsigned on = tile.on[jt];
        V a[NN];
        ap += n;
#pragma unroll
        for (int j = 0; j < NN; j++) {
            a[j] = an[j];
            if (mm + 1 < m1) an[j] = ap[node[j]];
        }
        if (!on) continue;
        // h_i = cff (g_i + sum_j g_j); sum_i h_i = cff (NN + 1) sum_j g_j
        typename LS::H hm[NN], hk[NN - 1];
        V sa = a[0];
#pragma unroll
        for (int j = 1; j < NN; j++) sa = vadd(sa, a[j]);
        hm[0] = LS::det(DIFF ? vscale(sa, cf0) : vscale(vadd(sa, a[0]), cff));
#pragma unroll
        for (int i = 1; i < NN; i++) hm[i] = LS::det(vscale(vadd(sa, a[i]), cff));
#pragma unroll
        for (int j = 1; j < NN; j++) a[j] = vsub(a[j], a[0]);
#pragma unroll
        for (int i = 0; i < NN - 1; i++) {
            V h = vscale(a[1], wdd[i][0]);
#pragma unroll
            for (int j = 1; j < NN - 1; j++) h = vadd(h, vscale(a[j + 1], wdd[i][j]));
            hk[i] = LS::det(h);
        }
#pragma unroll
        for (int g = 0; g < GQ; g++) {
            if (!(on >> g & 1)) continue;
            LS pm, pk;
#pragma unroll
            for (int i = NN - 1; i >= 0; i--) pm.add(f[g][i], hm[i]);
#pragma unroll
            for (int i = 0; i < NN - 1; i++) pk.add(DIFF ? f[g][i + 1] : LS::sub(f[g][i + 1], f[g][0]), hk[i]);
            const V y = tile.y[g][jt];
            put_link<V, JT>(j0, tile.row[g][jt], half, m.ne, vmul(pm.get(), y), vmul(pk.get(), y));
        }
    }
}

// The data gradient of toast's Gradient (GetGradient / AddDataGradient,
// src/python/toastmodule.cc:1745-1887).  Per link: with y = r + i i the
// linear projection, dn = 1/|y|^2, b = (data - model) / sd for the log
// amplitude and the phase (model = ln|y|, arg y), a = -2 b_mod / sd_mod and
// p = -2 b_arg / sd_arg, the detector vector enters the source's adjoint
// right-hand side twice: times (a r dn, -a i dn), then times (-p i dn, -p r dn).
__global__ void gradient_coef_kernel(int nqm, const cd* __restrict__ ylin, const cd* __restrict__ ylog,
                                     const double* __restrict__ data, const double* __restrict__ sd,
                                     cd* __restrict__ coef)
{
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= nqm) return;
    const double rp = ylin[l].x, ip = ylin[l].y, dn = 1.0 / (rp * rp + ip * ip);
    const double bm = (data[l] - ylog[l].x) / sd[l];
    const double ba = (data[nqm + l] - ylog[l].y) / sd[nqm + l];
    double t = -2.0 * bm / (1.0 * sd[l]);
    coef[2 * l] = cd{t * rp * dn, -t * ip * dn};
    t = -2.0 * ba / (1.0 * sd[nqm + l]);
    coef[2 * l + 1] = cd{-t * ip * dn, -t * rp * dn};
}

// adjoint right-hand sides w_q = sum over q's links (in order) of
// mvec_m coef1 + mvec_m coef2, written node-major in the solver's layout
__global__ void gradient_weights_kernel(int n, int nq, const cd* __restrict__ mvec, const int* __restrict__ link_ofs,
                                        const int* __restrict__ link_m, const cd* __restrict__ coef,
                                        const int* __restrict__ perm, cd* __restrict__ W)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y;
    if (i >= n || q >= nq) return;
    cd w = cd{0.0, 0.0};
    for (int l = link_ofs[q]; l < link_ofs[q + 1]; l++) {
        const cd r = mvec[(size_t)link_m[l] * n + i];
        w = vadd(w, vmul(r, coef[2 * l]));
        w = vadd(w, vmul(r, coef[2 * l + 1]));
    }
    W[(size_t)perm[i] * nq + q] = w;
}

// grad_mua[s] -= Re(f a), grad_kappa[s] -= Re(sum_d grad_d f grad_d a),
// summed over the sources in order (no voxel scaling); grad in/out
__global__ void gradient_accum_kernel(int dim, int slen, int nq, const cd* __restrict__ Pf, const cd* __restrict__ Pa,
                                      double* __restrict__ grad)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= slen) return;
    const int np = 1 + dim;
    double gm = grad[s], gk = grad[slen + s];
    for (int q = 0; q < nq; q++) {
        const cd* f = Pf + (size_t)q * np * slen + s;
        const cd* a = Pa + (size_t)q * np * slen + s;
        gm -= re(vmul(f[0], a[0]));
        cd k = cd{0.0, 0.0};
        for (int d = 1; d < np; d++) k = vadd(k, vmul(f[(size_t)d * slen], a[(size_t)d * slen]));
        gk -= re(k);
    }
    grad[s] = gm;
    grad[slen + s] = gk;
}

// Map_GridToSol (raster.cc:374-390) of Jacobian rows computed on the grid of
// a raster with an intermediate grid: row r of Jg (nb blocks of gslen grid
// points inside the mesh) -> row row0(r) of J (nb blocks of slen solution
// points): J[k] = sum over G's row of the solution point k of w Jg[col], in
// the row's entry order (RCompRowMatrix::Ax).  Rows r < half go to row0 + r,
// the others to row0 + r - half + hoff (the Im / kappa rows of a chunk of
// links).  add: J += instead of J = (the data gradient).  A thread per
// output entry.
template <class JT>
__global__ void grid_to_sol_rows_kernel(long long rows, int half, long long row0, long long hoff, int nb, int gslen,
                                        int slen, const int* __restrict__ rp, const int* __restrict__ col,
                                        const double* __restrict__ val, const JT* __restrict__ Jg,
                                        JT* __restrict__ J, int add)
{
    const long long total = rows * nb * (long long)slen;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(t % slen);
        const long long rb = t / slen;
        const int b = (int)(rb % nb);
        const long long r = rb / nb;
        const JT* x = Jg + (size_t)r * nb * gslen + (size_t)b * gslen;
        JT acc = (JT)0;
        for (int j = rp[k]; j < rp[k + 1]; j++) acc += (JT)val[j] * x[col[j]];
        const long long orow = r < half ? row0 + r : row0 + r - half + hoff;
        JT* y = J + (size_t)orow * nb * slen + (size_t)b * slen + k;
        *y = add ? *y + acc : acc;
    }
}

// Raster basis maps: y = A x row by row in entry order (RCompRowMatrix::Ax,
// crmatrix_imp.hpp:1168-1189; complex vectors component by component,
// Ax_cplx 1302-1327), one thread per (row, vector), `width` doubles per point.
// div (optional): each row's sum divided by div[row], 0 where that is 0 (a
// blob basis's node average, raster_bl.cc:170-204).
__global__ void csr_apply_kernel(int rows, int cols, int width, const int* __restrict__ rp,
                                 const int* __restrict__ col, const double* __restrict__ val,
                                 const double* __restrict__ x, double* __restrict__ y, const double* __restrict__ div)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x, v = blockIdx.y;
    if (r >= rows) return;
    const double* xv = x + (size_t)v * cols * width;
    for (int c = 0; c < width; c++) {
        double acc = 0.0;
        for (int j = rp[r]; j < rp[r + 1]; j++) acc = __dadd_rn(acc, __dmul_rn(val[j], xv[(size_t)col[j] * width + c]));
        if (div) acc = div[r] != 0.0 ? __ddiv_rn(acc, div[r]) : 0.0;
        y[((size_t)v * rows + r) * width + c] = acc;
    }
}

// basis -> solution points (Map_BasisToSol, raster.cc:292-315).  d: the
// pixel raster's real map D->Ax (raster_px.cc:147-150), 0 + 1 x, which
// turns -0 into +0
__global__ void gather_points_kernel(int slen, int glen, int width, const int* __restrict__ sol,
                                     const double* __restrict__ g, double* __restrict__ s, int d)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, v = blockIdx.y;
    if (i >= slen) return;
    for (int c = 0; c < width; c++) {
        const double x = g[((size_t)v * glen + sol[i]) * width + c];
        s[((size_t)v * slen + i) * width + c] = d ? __dadd_rn(0.0, x) : x;
    }
}

// solution points -> basis, zeros elsewhere (Map_SolToBasis, raster.cc:
// 318-345; d: the real D->ATx, 0 + 1 x)
__global__ void scatter_points_kernel(int slen, int glen, int width, const int* __restrict__ sol,
                                      const double* __restrict__ s, double* __restrict__ g, int d)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, v = blockIdx.y;
    if (i >= slen) return;
    for (int c = 0; c < width; c++) {
        const double x = s[((size_t)v * slen + i) * width + c];
        g[((size_t)v * glen + sol[i]) * width + c] = d ? __dadd_rn(0.0, x) : x;
    }
}

// QVec_Gaussian (src/libstoast/source.cc:19-56) for npos positions on the
// device: a thread per (node, position) gathers the contributions the
// reference scatters, in the reference's order (elements ascending, then the
// element's source nodes i ascending): q[js] += s_i BndIntFF(i, j) (Neumann:
// boundary source and receiving nodes only) or s_i IntFF(i, j), with
// s_i = exp(-d_i^2 / 2w^2) fac1.  scale (optional, n values) multiplies the
// result (detector vectors times c2a, toastmodule.cc:1189-1220).
__global__ void qvec_gaussian_kernel(int n, int dim, int nn, const double* __restrict__ coords,
                                     const int* __restrict__ el, const int* __restrict__ nel_ptr,
                                     const int* __restrict__ nel_list, const unsigned char* __restrict__ bnd,
                                     const double* __restrict__ intbff, const double* __restrict__ rec, int rec_len,
                                     int npos, const double* __restrict__ pos, double fac1, double fac2, int neumann,
                                     const double* __restrict__ scale, double* __restrict__ q)
{
    const int js = blockIdx.x * blockDim.x + threadIdx.x, p = blockIdx.y;
    if (js >= n || p >= npos) return;
    double acc = 0.0;
    if (!neumann || bnd[js]) {
        const double* c = pos + (size_t)p * dim;
        for (int t = nel_ptr[js]; t < nel_ptr[js + 1]; t++) {
            const int e = nel_list[t] >> 2, j = nel_list[t] & 3;
            const int* nd = el + (size_t)e * nn;
            for (int i = 0; i < nn; i++) {
                const int is = nd[i];
                if (neumann && !bnd[is]) continue;
                double d2 = 0.0;
                for (int k = 0; k < dim; k++) {
                    const double dk = c[k] - coords[(size_t)is * dim + k];
                    d2 += dk * dk;
                }
                const double d = sqrt(d2);
                const double sv = exp(d * d * fac2) * fac1;
                if (neumann) acc += sv * intbff[((size_t)e * nn + i) * nn + j];
                else acc += sv * ((i == j ? 2.0 : 1.0) * (dim == 2 ? 1.0 / 12.0 : 1.0 / 20.0) * rec[(size_t)e * rec_len]);
            }
        }
    }
    q[(size_t)p * n + js] = scale ? acc * scale[js] : acc;
}

}  // namespace tg
