// tg_direct.cuh -- the direct solver (LSOLVER_DIRECT): a multifrontal L D L^T
// factorisation in FP64 and its solves.
//
// The nested-dissection tree of the nodes (direct_pattern, tg_mesh.cu) gives
// one dense front per leaf block and per separator: its own nc columns and the
// nr rows of the ancestors that they touch, f = nc + nr, stored column by
// column (lower triangle).  The fronts of one height of the tree are
// independent and go through the same launches: assembly (entries of A and the
// children's update blocks), then per panel of DP columns one launch that
// factors the panel and one that updates the columns right of it.  Everything
// is deterministic: a front adds its children's blocks in their order.
//
// Why not the level-scheduled sparse kernels of the IC(0) sweeps: a complete
// factor has a level per column of the root path, 196 on the 3.2k-node disc,
// each a launch of a few rows with up to 150 serial merge steps (367 us a
// level).  The dense fronts turn that into about 70 launches (43 at the reset
// and 29 at the solve, with what surrounds them) bound by the FP64 rate (2 multiply-adds a clock on an SM): reset and 32 solves 60.0 -> 1.3 ms
// (3.2k nodes, 100 MHz), 337 -> 3.0 ms (12.5k nodes), 5.6 s -> 12.5 ms (7.5k-node
// cylinder).
//
// L D L^T and not L L^T: a column costs one reciprocal instead of a complex
// square root and a division, and the panels' diagonal blocks are the serial
// part.  Complex systems are complex symmetric; no pivoting, as before.
#pragma once
#include "tg_kernels.cuh"

namespace tg {

constexpr int DP = 16;     // panel columns
constexpr int DTR = 32;    // rows of a panel tile
constexpr int DKC = 8;     // right-hand sides per CTA of the solves

// 1 / d with two divisions (Smith's scaling for complex d)
__device__ __forceinline__ double direct_recip(double d) { return 1.0 / d; }
__device__ __forceinline__ cd direct_recip(cd d)
{
    if (fabs(d.x) >= fabs(d.y)) {
        const double r = d.y / d.x, t = 1.0 / fma(d.y, r, d.x);
        return cd{t, -r * t};
    }
    const double r = d.x / d.y, t = 1.0 / fma(d.x, r, d.y);
    return cd{r * t, -t};
}

// zero, the front's entries of A, and the children's update blocks; CTA =
// (front, part): the columns j with j % parts == part
template <class V>
__global__ void __launch_bounds__(256) direct_assemble_kernel(const DFront* __restrict__ fr, const int* __restrict__ ids,
                                                             const int* __restrict__ kids, const int* __restrict__ rel,
                                                             const DEntry* __restrict__ aent, const V* __restrict__ A,
                                                             V* vals)
{
    const DFront d = fr[ids[blockIdx.x]];
    const int part = blockIdx.y, parts = gridDim.y, f = d.nc + d.nr;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    V* F = vals + d.off;
    for (int j = part + warp * parts; j < f; j += nw * parts)
        for (int i = j + lane; i < f; i += 32) F[i + (size_t)j * f] = vzero<V>();
    __syncthreads();
    for (int e = threadIdx.x; e < d.na; e += blockDim.x) {
        const DEntry t = aent[d.a0 + e];
        if (t.j % parts == part) F[t.i + (size_t)t.j * f] = A[t.src];
    }
    for (int c = 0; c < d.nkid; c++) {
        __syncthreads();
        const DFront k = fr[kids[d.kid0 + c]];
        const int fk = k.nc + k.nr;
        const V* K = vals + k.off;
        const int* r = rel + k.rel0;
        for (int jc = warp; jc < k.nr; jc += nw) {
            const int J = r[jc];
            if (J % parts != part) continue;
            V* col = F + (size_t)J * f;
            const V* src = K + k.nc + (size_t)(k.nc + jc) * fk;
            for (int ic = jc + lane; ic < k.nr; ic += 32) col[r[ic]] = vadd(col[r[ic]], src[ic]);
        }
    }
}

// Panel of columns [p0, p0 + nb): every CTA factors the DP x DP diagonal block
// (a launch and a round trip through memory less than a CTA that does it for
// the others) and forms its tile of DTR rows below: l_ij = w_ij / d_j with
// w_ij = a_ij - sum_t w_it l_jt.  Tile 0 writes the block (unit L below, d on
// the diagonal) to blk, DP values per column rank, and 1 / d; the front itself
// keeps the block's input, which the other CTAs may still be reading.
template <class V>
__global__ void __launch_bounds__(128) direct_panel_kernel(const DFront* __restrict__ fr, const int* __restrict__ ids,
                                                          int p0, V* vals, V* __restrict__ blk,
                                                          V* __restrict__ dinv)
{
    __shared__ V D[DP][DP + 1];    // D[i][j], j <= i: w before, l after its column's step
    __shared__ V di[DP];
    const DFront d = fr[ids[blockIdx.x]];
    if (p0 >= d.nc) return;
    const int f = d.nc + d.nr, nb = min(DP, d.nc - p0), r0 = p0 + nb + blockIdx.y * DTR;
    if (blockIdx.y > 0 && r0 >= f) return;
    const int tid = threadIdx.x;
    V* F = vals + d.off;
    for (int e = tid; e < nb * nb; e += blockDim.x) {
        const int i = e % nb, j = e / nb;
        if (i >= j) D[i][j] = F[(p0 + i) + (size_t)(p0 + j) * f];
    }
    // this thread's row of the tile, in flight during the factorisation
    const int row = r0 + tid;
    const bool have = tid < DTR && row < f;
    V w[DP];
#pragma unroll
    for (int j = 0; j < DP; j++) w[j] = have && j < nb ? F[row + (size_t)(p0 + j) * f] : vzero<V>();
    __syncthreads();
    for (int j = 0; j < nb; j++) {
        if (tid == 0) di[j] = direct_recip(D[j][j]);
        __syncthreads();
        const V r = di[j];
        // columns right of j: a_ik -= w_ij l_kj
        for (int e = tid; e < DP * DP; e += blockDim.x) {
            const int i = e % DP, k = e / DP;
            if (k > j && i >= k && i < nb) D[i][k] = vfms(D[i][k], D[i][j], vmul(D[k][j], r));
        }
        __syncthreads();
        if (tid > j && tid < nb) D[tid][j] = vmul(D[tid][j], r);
    }
    __syncthreads();
    if (blockIdx.y == 0) {
        for (int e = tid; e < nb * nb; e += blockDim.x) {
            const int i = e % nb, j = e / nb;
            if (i >= j) blk[(size_t)(d.c0 + p0 + i) * DP + j] = D[i][j];
        }
        if (tid < nb) dinv[d.c0 + p0 + tid] = di[tid];
    }
    if (!have) return;
#pragma unroll
    for (int j = 0; j < DP; j++) {
        if (j >= nb) break;
#pragma unroll
        for (int t = 0; t < DP; t++)
            if (t < j) w[j] = vfms(w[j], w[t], D[j][t]);
        F[row + (size_t)(p0 + j) * f] = vmul(w[j], di[j]);
    }
}

// The columns right of the panel: C_ik -= sum_j l_ij d_j l_kj, a CTA per
// DP x DP tile of the lower triangle (tiles counted row by row)
template <class V>
__global__ void __launch_bounds__(DP * DP) direct_update_kernel(const DFront* __restrict__ fr,
                                                               const int* __restrict__ ids, int p0, int t0,
                                                               const V* __restrict__ blk, V* vals)
{
    __shared__ V L[DP][DP + 1], K[DP][DP + 1];  // [j][row]
    const DFront d = fr[ids[blockIdx.x]];
    if (p0 >= d.nc) return;
    const int f = d.nc + d.nr, nb = min(DP, d.nc - p0), c0 = p0 + nb;
    const int nt = (f - c0 + DP - 1) / DP;
    const long long t = (long long)t0 + blockIdx.y;
    if (t >= (long long)nt * (nt + 1) / 2) return;
    int ti = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
    while ((long long)(ti + 1) * (ti + 2) / 2 <= t) ti++;
    while ((long long)ti * (ti + 1) / 2 > t) ti--;
    const int tj = (int)(t - (long long)ti * (ti + 1) / 2);
    V* F = vals + d.off;
    const int x = threadIdx.x % DP, y = threadIdx.x / DP;
    const int ri = c0 + ti * DP + x, rk = c0 + tj * DP + x;
    if (y < nb) {
        const V dj = blk[(size_t)(d.c0 + p0 + y) * DP + y];
        L[y][x] = ri < f ? F[ri + (size_t)(p0 + y) * f] : vzero<V>();
        K[y][x] = rk < f ? vmul(F[rk + (size_t)(p0 + y) * f], dj) : vzero<V>();
    }
    __syncthreads();
    const int k = c0 + tj * DP + y;
    if (ri >= f || k >= f || k > ri) return;
    V acc = F[ri + (size_t)k * f];
    for (int j = 0; j < nb; j++) acc = vfms(acc, L[j][x], K[j][y]);
    F[ri + (size_t)k * f] = acc;
}

// Forward solve of a front: w = [b of its columns; 0] plus the children's
// parts, y = L^-1 w on its columns (to X), the rest stays in w for its parent.
// CTA = (front of nf, DKC right-hand sides), in one grid dimension; w: [front
// rows][k].
template <class V>
__global__ void __launch_bounds__(256) direct_fwd_kernel(const DFront* __restrict__ fr, const int* __restrict__ ids,
                                                        const int* __restrict__ kids, const int* __restrict__ rel,
                                                        const int* __restrict__ rows, const V* __restrict__ vals,
                                                        const V* __restrict__ blk, int nf, int k, const V* __restrict__ B,
                                                        V* X, V* W)
{
    const DFront d = fr[ids[blockIdx.x % nf]];
    const int f = d.nc + d.nr, c0 = blockIdx.x / nf * DKC, kc = min(DKC, k - c0), tid = threadIdx.x, nt = blockDim.x;
    const V* F = vals + d.off;
    V* w = W + (size_t)d.w0 * k + c0;
    const int* rw = rows + d.w0;
    for (int e = tid; e < f * kc; e += nt) {
        const int i = e / kc, c = e % kc;
        w[(size_t)i * k + c] = i < d.nc ? B[(size_t)rw[i] * k + c0 + c] : vzero<V>();
    }
    for (int q = 0; q < d.nkid; q++) {
        __syncthreads();
        const DFront s = fr[kids[d.kid0 + q]];
        const V* ws = W + ((size_t)s.w0 + s.nc) * k + c0;
        const int* r = rel + s.rel0;
        for (int e = tid; e < s.nr * kc; e += nt) {
            const int i = e / kc, c = e % kc;
            V* o = w + (size_t)r[i] * k + c;
            *o = vadd(*o, ws[(size_t)i * k + c]);
        }
    }
    for (int p0 = 0; p0 < d.nc; p0 += DP) {
        const int nb = min(DP, d.nc - p0);
        __shared__ V y[DP][DKC], D[DP][DP + 1];
        __syncthreads();
        for (int e = tid; e < nb * DP; e += nt) D[e / DP][e % DP] = blk[(size_t)(d.c0 + p0) * DP + e];
        for (int e = tid; e < nb * kc; e += nt) y[e / kc][e % kc] = w[(size_t)(p0 + e / kc) * k + e % kc];
        __syncthreads();
        for (int j = 0; j < nb; j++) {
            const int i = tid / DKC, c = tid % DKC;
            if (i > j && i < nb && c < kc) y[i][c] = vfms(y[i][c], D[i][j], y[j][c]);
            __syncthreads();
        }
        for (int e = tid; e < nb * kc; e += nt) X[(size_t)rw[p0 + e / kc] * k + c0 + e % kc] = y[e / kc][e % kc];
        // rows below the panel
        const int m = f - p0 - nb;
        for (int e = tid; e < m * DKC; e += nt) {
            const int i = e / DKC, c = e % DKC;
            if (c >= kc) continue;
            V* o = w + (size_t)(p0 + nb + i) * k + c;
            V acc = *o;
            const V* l = F + (p0 + nb + i) + (size_t)p0 * f;
#pragma unroll 8
            for (int j = 0; j < nb; j++) acc = vfms(acc, l[(size_t)j * f], y[j][c]);
            *o = acc;
        }
    }
}

// Backward solve: x = L^-T D^-1 y on the front's columns, given x at its rows
template <class V>
__global__ void __launch_bounds__(256) direct_bwd_kernel(const DFront* __restrict__ fr, const int* __restrict__ ids,
                                                        const int* __restrict__ rows, const V* __restrict__ vals,
                                                        const V* __restrict__ blk, const V* __restrict__ dinv, int nf,
                                                        int k,
                                                        V* X, V* W)
{
    const DFront d = fr[ids[blockIdx.x % nf]];
    const int f = d.nc + d.nr, c0 = blockIdx.x / nf * DKC, kc = min(DKC, k - c0), tid = threadIdx.x, nt = blockDim.x;
    const V* F = vals + d.off;
    V* w = W + (size_t)d.w0 * k + c0;
    const int* rw = rows + d.w0;
    for (int e = tid; e < f * kc; e += nt) {
        const int i = e / kc, c = e % kc;
        const V v = X[(size_t)rw[i] * k + c0 + c];
        w[(size_t)i * k + c] = i < d.nc ? vmul(v, dinv[d.c0 + i]) : v;
    }
    const int np = (d.nc + DP - 1) / DP;
    for (int p = np - 1; p >= 0; p--) {
        const int p0 = p * DP, nb = min(DP, d.nc - p0);
        __shared__ V y[DP][DKC], part[DP][DKC], D[DP][DP + 1];
        __syncthreads();
        for (int e = tid; e < nb * DP; e += nt) D[e / DP][e % DP] = blk[(size_t)(d.c0 + p0) * DP + e];
        // y_j = w_j - sum over the rows below the panel: a thread per column j,
        // right-hand side c and half of the rows
        const int c = tid % DKC, j = tid / DKC % DP, h = tid / (DKC * DP);
        V acc = vzero<V>();
        if (j < nb && c < kc) {
            const V* l = F + (size_t)(p0 + j) * f;
#pragma unroll 4
            for (int i = p0 + nb + h; i < f; i += 2) acc = vfma(acc, l[i], w[(size_t)i * k + c]);
            if (h) part[j][c] = acc;
        }
        __syncthreads();
        if (h == 0 && j < nb && c < kc) y[j][c] = vsub(w[(size_t)(p0 + j) * k + c], vadd(acc, part[j][c]));
        __syncthreads();
        for (int j = nb - 1; j >= 0; j--) {
            const int i = tid / DKC;
            if (i < j && c < kc) y[i][c] = vfms(y[i][c], D[j][i], y[j][c]);
            __syncthreads();
        }
        for (int e = tid; e < nb * kc; e += nt) {
            const int i = e / kc, c = e % kc;
            w[(size_t)(p0 + i) * k + c] = y[i][c];
            X[(size_t)rw[p0 + i] * k + c0 + c] = y[i][c];
        }
    }
}

}  // namespace tg
