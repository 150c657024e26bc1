// tg_cluster.cuh -- the interface of the resident solve (tg_resident.cu): one
// kernel in which thread-block clusters run a conjugate-gradient process on
// their own right-hand sides, and the kernel that forms its preconditioner.
#pragma once
#include "tg_kernels.cuh"

namespace tg {

constexpr int CL_NT = 800;      // threads per CTA at most (80 registers each)
constexpr int CL_MAXCG = 4;     // columns per cluster at most
constexpr int CL_MAXCS = 16;    // CTAs per cluster at most
constexpr int CL_NV = 3;        // quantities per column in one reduction at most
constexpr int FSAI_MAXM = 32;   // entries of a row of G at most

// a matrix in slices of 32 rows, entry by entry: entry e of row r at
// ptr[r / 32] + 32 e + r % 32, its column as the slot of the CTA's gather
// buffers; padding: the row's own slot and the value 0
template <class V>
struct Sell {
    const int* ptr;
    const unsigned short* col;
    const V* val;
};

template <class V64, class V32>
struct ResArgs {
    int n, k, cs;
    int slots;                  // rows of a gather buffer (own rows and halo), the largest of the CTAs
    int msm, mofs_val, mofs_col, mofs_ptr, mofs_push;  // msm: the matrices go to shared memory, at these byte offsets
    Sell<V32> A, G, T;          // system matrix, approximate inverse and its transpose
    const int* pofs;            // per CTA: its halo copies in push,
    const uint2* push;          //   {own slot, rank << 16 | slot there}
    V32* x;                     // FP32 correction, [cluster][node][CG]
    V64 *X, *R;                 // solution and true residual, node-major, k columns
    const V64* B;
    void* Xff;                  // solution of the columns being updated, as float-float, node-major
    const int *rowptr, *colidx; // layout CSR of the system matrix, for the residuals:
    const V64* A64;             //   FP64 values,
    const void* Aff;            //   float-float values,
    const float* absA;          //   magnitudes
    ColState* co;               // per column: tol on entry, results on exit
    float trig;                 // residual drop that triggers a correction
    double cwtol;               // componentwise bound (0: none)
    int maxit, max_upd, zero_guess;
    int per;                    // iterations that a result counts as one
    int all64;                  // every residual product in FP64
};

// the kernel for lv columns a cluster (1, 2; real systems also 4)
template <class V64, class V32>
void (*resident_kernel(int lv))(ResArgs<V64, V32>);

// Both sweeps of the IC(0) apply in one launch: a cluster per lv columns
template <class V>
struct IcClArgs {
    IcSweepDev f, b;
    const V *vf, *vb;           // entries of the factor in the sweeps' layouts
    const V* dinv;
    const V* in;                // right-hand sides, node-major, k columns
    V* out;                     // result
    int n, k, cs;
    int mofs;                   // byte offset of the levels and rows in shared memory
    const ColState* st;         // columns with active != 1 keep their values (null: all)
};
constexpr int IC_NT = 256;      // threads of a CTA
template <class V>
void (*ic_cluster_kernel_of(int lv))(IcClArgs<V>);

// G of the approximate inverse from A's float-float values in CSR order; the first n32 CTAs
// take the rows of 17 to 32 entries, the next n16 those of 9 to 16, the others
// those of at most 8
constexpr int FSAI_NT = 128;
constexpr int fsai_rows(int gl) { return gl == 32 ? 2 : FSAI_NT / gl; }  // rows of such a CTA (35 KB of complex matrices)
template <class V64, class V>
void (*fsai_kernel_of())(int n, int n32, int n16, const int* rowptr, const int* colidx, const int* diagpos, const void* A,
                         const int* gptr, const int* gcol, const int* gcnt, V* gval);

}  // namespace tg
