// Static (implicit) solver on the GPU: displacement-controlled Newton-Raphson
// after solvers/scripts/static/newtonraphsondisplacementcontrolled.m, with the
// tangent of buildstiffnessmatrixCSCformat.m solved matrix-free by a
// block-Jacobi preconditioned conjugate gradient over the free DOFs.
//
// One load step: the prescribed DOFs move by the increment, then each Newton
// iteration
//   1. updates every bond from the current positions (calculatedeformedlength,
//      the softening law, calculatebondfailure with the law's sc) and forms the
//      bond forces of calculatebondforces.m (BFMULTIPLIER included, unlike the
//      MEX) and their serial nodal sum in bond order (calculatenodalforces.m),
//      times cellVolume as the driver does (:111);
//   2. stops when the out-of-balance force on the free DOFs is at most `tol`
//      times the force on the held DOFs (the reference compares with 0.5 % of
//      the net internal force, checkconvergencecriteria.m:21-29);
//   3. solves K delta = F on the free DOFs, K the sum over intact bonds of
//      rig [c c^T, -c c^T; -c c^T, c c^T] with rig = BFM (BS / L^3) VCF V^2
//      (1 - BSF) at the current bond vector c (buildstiffnessmatrixCSCformat.m
//      NOD = 3 branch), and moves the free nodes by delta.
// The reference solves with MATLAB's bicgstabl and lsqr and applies its own
// corrector conventions; here every linear solve is a PCG to a relative
// residual of cg_tol, so results agree with a direct solve of the same
// equations to that tolerance.
//
// Layout: per bond its end nodes, constants and state; per node the list of
// its bond ends in bond order (a stable radix sort of the directed entries by
// node), which gives the nodal sums their serial order. For the matrix-free
// products the lists are also laid out in slices of 32 nodes, entry k of the
// slice's 32 lists side by side (padded to its longest list): the neighbour's id
// and, per tangent, the bond's stiffness scale, 12 bytes an entry. Where padding would
// take most of that (a few nodes with very long lists) they stay lists. The bond
// vector is the difference of the two nodes' positions, which lie in one record
// with the direction p. Reductions are fixed-order, so a step is deterministic.
#include "bbpd_internal.h"
#include "gridbarrier.cuh"
#include "nodalsum.cuh"
#include "physics.cuh"
#include "staging.cuh"

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cmath>
#include <memory>
#include <vector>

using namespace bbpd;

namespace {

constexpr int kThreads = 256;
constexpr int kRedBlocks = 592;   // partial-sum blocks of the dot products (4 per SM)

inline int blocks_for(int64_t n)
{
    int64_t b = (n + kThreads - 1) / kThreads;
    return (int)std::max<int64_t>(1, std::min<int64_t>(b, 148 * 64));
}

#define GRID_STRIDE(i, n) \
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

#define TRY(x) do { int r_ = (x); if (r_) return r_; } while (0)

int launch_check()
{
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(BBPD_ERR_CUDA, "kernel launch: %s", cudaGetErrorString(e));
    return BBPD_OK;
}

struct SBonds {
    const uint32_t *a, *b;      // end nodes (0-based)
    const double *L0, *BS, *VCF, *BFM;
    const uint8_t *BT;
    double *fail, *bsf;
    uint8_t *flag;
    double *rig;                // tangent scale, 0 for failed bonds
    double *f;                  // bond force, [3 nB]
    int64_t nB;
    int law;
    LawScalars P;
    double V;
};

// calculatedeformedlength + law + calculatebondfailure + calculatebondforces.m
// and the stiffness scale of buildstiffnessmatrixCSCformat.m for every bond
__global__ void k_static_bonds(SBonds s, const double *__restrict__ x, int64_t n)
{
    GRID_STRIDE(k, s.nB)
    {
        const int64_t i = s.a[k], j = s.b[k];
        double dX, dY, dZ, L, st;
        bond_kinematics(x[i], x[i + n], x[i + 2 * n], x[j], x[j + n], x[j + 2 * n], s.L0[k], dX, dY, dZ, L, st);
        double B = s.bsf[k], fl = s.fail[k];
        bool soft = s.flag[k] != 0;
        const int bt = s.BT[k];
        if (s.law == BBPD_LAW_BILINEAR) {
            double f = soft ? 1.0 : 0.0;
            if (bt == 0 && st > s.P.s0) f = 1;
            const double bs = ((st - s.P.s0) / st) * (s.P.sc / (s.P.sc - s.P.s0));
            B = matlab_max(B, bs * f);
            if (B > 1) B = 1;
            if (isnan(B)) B = 0;
            soft = f != 0;
        } else if (s.law == BBPD_LAW_TRILINEAR) {
            law_trilinear(st, s.P.s0, s.P.s1, s.P.sc, s.P, false, bt == 0, B, soft);
        } else if (s.law == BBPD_LAW_EXPONENTIAL) {
            law_exponential(st, s.P.s0, s.P.sc, s.P, bt == 0, B, soft);
        }
        law_linear(st, s.P.sc, s.P, bt, fl);
        s.bsf[k] = B;
        s.fail[k] = fl;
        s.flag[k] = soft ? 1 : 0;
        const double t = s.BFM[k] * fl * s.BS[k] * (1 - B) * st * s.V * s.VCF[k];
        const double d[3] = {dX, dY, dZ};
        for (int c = 0; c < 3; c++) {
            double f = t * (d[c] / L);
            if (f != f) f = 0.0;
            s.f[k + c * s.nB] = f;
        }
        // rig = BFM * ((BS / L^3) * VCF * V^2) * (1 - BSF) for intact bonds
        const double r = fl == 1 ? s.BFM[k] * ((s.BS[k] / (L * L * L)) * s.VCF[k] * (s.V * s.V)) * (1 - B) : 0.0;
        s.rig[k] = isfinite(r) ? r : 0.0;
    }
}

struct SNodes {
    const int64_t *off;         // [n + 1] list offsets
    const uint32_t *ent;        // directed entries q = 2k + side, by node, in bond order
    const int64_t *sptr;        // slots of slice s: [sptr[s], sptr[s + 1]), 32 a row
    const uint32_t *bond, *col; // bond and neighbour of every slot (LISTS: of every list entry)
    int64_t ns;
    const uint8_t *held;        // per DOF [3 n]: 1 support, 2 prescribed
    int64_t n, nB;
};

// calculatenodalforces.m:25-35 in its serial order (node i gets +f of the bonds
// it starts, -f of those it ends), times cellVolume (driver :111); the residual
// norms of the free and held DOFs go to per-block partial sums.
__global__ void __launch_bounds__(kThreads) k_static_nodal(SNodes g, const double *__restrict__ f, double V, double *F,
                                                           double *part)
{
    __shared__ NodeSumShared sm[kThreads / 32];
    __shared__ double sh[2][kThreads / 32];
    double rf = 0, rh = 0;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t warps = (int64_t)gridDim.x * (kThreads / 32);
    for (int64_t k = (int64_t)blockIdx.x * (kThreads / 32) + w; k * kNodes < g.n; k += warps) {
        const int64_t i = k * kNodes + lane / 3, e = i + (lane % 3) * g.n;
        double t = 0.0, a;
        warp_node_sums<false>(g.off, g.ent, k * kNodes, g.n, f, f + g.nB, f + 2 * g.nB, sm[w], t, a);
        if (lane < 3 * kNodes && i < g.n) {
            const double v = a * V;
            F[e] = v;
            if (g.held[e]) rh += v * v;
            else rf += v * v;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        rf += __shfl_xor_sync(0xffffffffu, rf, o);
        rh += __shfl_xor_sync(0xffffffffu, rh, o);
    }
    if (lane == 0) {
        sh[0][w] = rf;
        sh[1][w] = rh;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double s0 = 0, s1 = 0;
        for (int q = 0; q < kThreads / 32; q++) {
            s0 += sh[0][q];
            s1 += sh[1][q];
        }
        part[2 * blockIdx.x] = s0;
        part[2 * blockIdx.x + 1] = s1;
    }
}

// The slices: length of each (its longest list), times 32 for the scan
__global__ void k_slice_lengths(const int64_t *__restrict__ off, int64_t n, int64_t ns, int64_t *cnt)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; s <= ns; s += warps) {
        const int64_t i = s * 32 + lane;
        int len = s < ns && i < n ? (int)(off[i + 1] - off[i]) : 0;
        for (int o = 16; o > 0; o >>= 1) len = max(len, __shfl_xor_sync(0xffffffffu, len, o));
        if (lane == 0) cnt[s] = (int64_t)len * 32;
    }
}

constexpr uint32_t kNoBond = 0xFFFFFFFFu;

// Bond and neighbour of every slot; padding names the node itself and no bond
__global__ void k_slice_fill(const int64_t *__restrict__ off, const uint32_t *__restrict__ ent,
                             const uint32_t *__restrict__ a, const uint32_t *__restrict__ b, int64_t n, int64_t ns,
                             const int64_t *__restrict__ sptr, uint32_t *bond, uint32_t *col)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; s < ns; s += warps) {
        const int64_t i = s * 32 + lane, e0 = i < n ? off[i] : 0, e1 = i < n ? off[i + 1] : 0;
        const int64_t len = (sptr[s + 1] - sptr[s]) >> 5;
        for (int64_t k = 0; k < len; k++) {
            const int64_t at = sptr[s] + k * 32 + lane;
            uint32_t q = kNoBond, j = i < n ? (uint32_t)i : 0u;
            if (e0 + k < e1) {
                const uint32_t v = ent[e0 + k];
                q = v >> 1;
                j = (v & 1u) ? a[q] : b[q];
            }
            bond[at] = q;
            col[at] = j;
        }
    }
}

// The same for lists that stay lists
__global__ void k_list_fill(const uint32_t *__restrict__ ent, const uint32_t *__restrict__ a, const uint32_t *__restrict__ b,
                            int64_t m, uint32_t *bond, uint32_t *col)
{
    GRID_STRIDE(e, m)
    {
        const uint32_t v = ent[e], q = v >> 1;
        bond[e] = q;
        col[e] = (v & 1u) ? a[q] : b[q];
    }
}

// A node's position and its component of the CG direction p (zero on held and
// left-out DOFs): 64 bytes, read as a 256-bit and a 128-bit load
struct __align__(64) NodeRec {
    double x, y, z, px, py, pz, pad[2];
};
struct Rec6 {
    double x, y, z, px, py, pz;
};

__device__ __forceinline__ Rec6 load_rec(const NodeRec *p)
{
    Rec6 r;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.px) : "l"(p));
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(r.py), "=d"(r.pz) : "l"(&p->py));
    return r;
}

// What a linear solve reads: position records, every slot's stiffness scale,
// and the block-Jacobi preconditioner: the inverse of each node's 3 x 3
// diagonal block restricted to its free DOFs (symmetric, 6 values); a DOF
// without stiffness (every bond of its node broken) is left out of the solve.
__global__ void k_static_records(const double *__restrict__ x, int64_t n, NodeRec *rec)
{
    GRID_STRIDE(i, n)
    {
        rec[i].x = x[i];
        rec[i].y = x[i + n];
        rec[i].z = x[i + 2 * n];
    }
}

__global__ void k_slot_rig(const uint32_t *__restrict__ bond, const double *__restrict__ rig,
                           int64_t entries, double *rigE)
{
    GRID_STRIDE(e, entries)
    {
        const uint32_t q = bond[e];
        rigE[e] = q == kNoBond ? 0.0 : rig[q];
    }
}

// A lane adds its node's list in bond order, four rows of the slice in flight.
template <bool LISTS>
__global__ void k_static_precond(SNodes g, const double *__restrict__ rigE, const NodeRec *__restrict__ rec, double *Minv,
                                 uint8_t *skip)
{
    const int64_t n = g.n;
    GRID_STRIDE(i, n)
    {
        const int64_t s = i >> 5, rows = LISTS ? g.off[i + 1] - g.off[i] : (g.sptr[s + 1] - g.sptr[s]) >> 5;
        const int64_t at = LISTS ? g.off[i] : g.sptr[s] + (i & 31);
        constexpr int kRow = LISTS ? 1 : 32;
        const uint32_t *col = g.col + at;
        const double *rig = rigE + at;
        const double xi[3] = {rec[i].x, rec[i].y, rec[i].z};
        double D[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
#pragma unroll 4
        for (int64_t k = 0; k < rows; k++) {
            const double r = rig[k * kRow];
            const NodeRec *o = rec + col[k * kRow];
            const double c[3] = {o->x - xi[0], o->y - xi[1], o->z - xi[2]};
            for (int u = 0; u < 3; u++)
                for (int v = 0; v < 3; v++) D[u][v] += r != 0 ? r * c[u] * c[v] : 0.0;
        }
        bool fr[3];
        for (int u = 0; u < 3; u++) {
            fr[u] = !g.held[i + u * n] && D[u][u] > 0;
            skip[i + u * n] = fr[u] ? 0 : 1;
        }
        for (int u = 0; u < 3; u++)
            for (int v = 0; v < 3; v++)
                if (!fr[u] || !fr[v]) D[u][v] = (u == v) ? 1.0 : 0.0;
        // inverse of the symmetric 3 x 3 block by cofactors
        const double c00 = D[1][1] * D[2][2] - D[1][2] * D[2][1];
        const double c01 = D[1][2] * D[2][0] - D[1][0] * D[2][2];
        const double c02 = D[1][0] * D[2][1] - D[1][1] * D[2][0];
        const double det = D[0][0] * c00 + D[0][1] * c01 + D[0][2] * c02;
        double m[6];
        if (det > 0 && isfinite(det)) {
            const double id = 1.0 / det;
            m[0] = c00 * id;
            m[1] = c01 * id;
            m[2] = c02 * id;
            m[3] = (D[0][0] * D[2][2] - D[0][2] * D[2][0]) * id;
            m[4] = (D[0][2] * D[1][0] - D[0][0] * D[1][2]) * id;
            m[5] = (D[0][0] * D[1][1] - D[0][1] * D[1][0]) * id;
        } else {   // degenerate block: scalar Jacobi
            m[0] = 1.0 / D[0][0];
            m[3] = 1.0 / D[1][1];
            m[5] = 1.0 / D[2][2];
            m[1] = m[2] = m[4] = 0.0;
        }
        for (int q = 0; q < 6; q++) Minv[i + q * n] = m[q];
    }
}

__device__ __forceinline__ void apply_minv(const double m[6], const double r[3], double z[3])
{
    z[0] = m[0] * r[0] + m[1] * r[1] + m[2] * r[2];
    z[1] = m[1] * r[0] + m[3] * r[1] + m[4] * r[2];
    z[2] = m[2] * r[0] + m[4] * r[1] + m[5] * r[2];
}

// Sum of `w` interleaved partial streams of `nb` blocks to out[0..w): one warp
// per stream, lanes 32 apart, then the butterfly
__global__ void k_reduce(const double *__restrict__ part, int nb, int w, double *out)
{
    const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
    if (k >= w) return;
    double s = 0;
    for (int b = lane; b < nb; b += 32) s += part[b * w + k];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) out[k] = s;
}

constexpr int kCgThreads = 512;   // 16 warps of 128 registers on every SM
constexpr int kCgWarps = kCgThreads / 32;
constexpr int kCgRows = 4;         // rows of a warp's gathers in flight
constexpr int kCgCheck = 8;        // iterations between convergence checks
constexpr int kCgLaunch = 1024;    // iterations of one launch at most (bbpd_selftest_static_launch changes it)
// The sums keep the order of 592 groups of 8 warps, whatever the grid: p.Kp goes
// over the nodes warp by warp (lane l of owner o stands for warp 32 o + l, which
// takes nodes 32 o + l, 32 o + l + 4736, ...), r.z and r.r over them 32 at a time.
constexpr int kCgGroups = 592;
constexpr int kCgOwners = kCgGroups / 4;
constexpr int kCgSlices = 5;       // slices a block multiplies between two syncs: 15 sums for its 16 warps

struct CgShared {
    double acc[kCgSlices][kCgWarps][3][32];   // K p: two of a node's 32 partial sums, folded
    double py[kCgSlices][3][32];              // p_c (K p)_c
    double2 part[kCgGroups];
    double sh[2][kCgWarps];
    double2 sum;
};

// The grid's two sums: every block adds the groups' partials for itself, in
// group order, after the barrier.
__device__ __forceinline__ double2 add_groups(const double2 *part, int count, CgShared &sm)
{
    for (int k = threadIdx.x; k < count; k += kCgThreads) sm.part[k] = __ldcg(&part[k]);
    __syncthreads();
    if (threadIdx.x == 0) {
        double u = 0;
#pragma unroll 8
        for (int k = 0; k < count; k++) u += sm.part[k].x;
        sm.sum.x = u;
    } else if (threadIdx.x == 32) {
        double v = 0;
#pragma unroll 8
        for (int k = 0; k < count; k++) v += sm.part[k].y;
        sm.sum.y = v;
    }
    __syncthreads();
    return sm.sum;
}

struct CgArgs {
    SNodes g;
    const double *rigE;            // stiffness scale of every slot (0: failed bond or padding)
    NodeRec *rec;
    const double *F, *Minv;
    const uint8_t *skip;
    double *x;                     // moved by the solution once the solve ends
    double *d, *r, *z;
    double *y;                     // K p
    double2 *part;                 // 2 x kCgGroups partials
    double *scal;                  // [0] r.z, [1] r.r, [2] r.r at the start
    int *state;                    // [0] CG_*, [1] iterations so far, [2] error word
    unsigned *bar;
    unsigned long long timeout_ns;
    double tol2;                   // stop at r.r <= tol2 * r.r at the start
    int first, max_cg, launch;     // launch: iterations of this launch at most
};
enum { CG_MORE = 0, CG_DONE = 1, CG_NONFINITE = 2 };

// r.z and r.r of all nodes: node(i, rz, rr) does a node's work and adds its terms.
// A warp takes 32 nodes, 8 warps a group; sums over the warp, then the group.
template <class F>
__device__ __forceinline__ void node_sums(int64_t n, double2 *part, CgShared &sm, F node)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int groups = (int)min((int64_t)kCgGroups, (n + 255) / 256);
    for (int v0 = 0; v0 < groups; v0 += 2 * gridDim.x) {
        const int v = v0 + blockIdx.x + (w >> 3) * gridDim.x;
        double rz = 0, rr = 0;
        if (v < groups)
            for (int64_t i = 256 * (int64_t)v + 32 * (w & 7) + lane; i < n; i += 256 * (int64_t)kCgGroups) node(i, rz, rr);
        for (int o = 16; o > 0; o >>= 1) {
            rz += __shfl_xor_sync(0xffffffffu, rz, o);
            rr += __shfl_xor_sync(0xffffffffu, rr, o);
        }
        __syncthreads();   // sh is free
        if (lane == 0) {
            sm.sh[0][w] = rz;
            sm.sh[1][w] = rr;
        }
        __syncthreads();
        if ((threadIdx.x & 255) == 0 && v < groups) {
            double2 s = make_double2(0, 0);
            for (int k = 0; k < 8; k++) {
                s.x += sm.sh[0][w + k];
                s.y += sm.sh[1][w + k];
            }
            part[v] = s;
        }
    }
}

// y = K p of the owners' slices (slice s belongs to owner s mod kCgOwners) and the
// partials of p.y. A node's sum is 32 partial sums (entries l, l + 32, ... to
// partial l) folded in a butterfly; warp w of the block takes partials w and
// w + 16 of the slice's 32 nodes.
template <bool LISTS>
__device__ __forceinline__ void cg_product(const SNodes &g, const double *rigE, const NodeRec *rec, double *y, double2 *part,
                                           CgShared &sm)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t n = g.n;
    for (int own = blockIdx.x; own < kCgOwners && own < g.ns; own += gridDim.x) {
        const int64_t count = (g.ns - own + kCgOwners - 1) / kCgOwners;
        double acc = 0;   // warp 0: p.y of the warp this lane stands for
        for (int64_t m = 0; m < count; m += kCgSlices) {
            const int G = (int)min((int64_t)kCgSlices, count - m);
            // lane k < G holds the place and rows of slice k
            int64_t at = 0;
            int len = 0;
            if (lane < G) {
                const int64_t s = own + kCgOwners * (m + lane);
                at = g.sptr[s];
                len = (int)((g.sptr[s + 1] - at) >> 5);
            }
            uint32_t j[kCgRows];
            double h[kCgRows];
            // rows k, k + 32, ... of slice q, if it has them: neighbours and scales
            auto streams = [&](int q, int k) {
                int64_t b;
                int rows;
                constexpr int64_t kRow = LISTS ? 1 : 32;
                if (LISTS) {
                    const int64_t i = (own + kCgOwners * (m + q)) * 32 + lane;
                    b = i < n ? g.off[i] : 0;
                    rows = i < n ? (int)(g.off[i + 1] - b) : 0;
                } else {
                    b = __shfl_sync(0xffffffffu, at, q) + lane;
                    rows = __shfl_sync(0xffffffffu, len, q);
                }
#pragma unroll
                for (int t = 0; t < kCgRows; t++) {
                    const int row = k + 32 * t;
                    j[t] = row < rows ? __ldg(g.col + b + row * kRow) : 0u;
                    h[t] = row < rows ? __ldg(rigE + b + row * kRow) : 0.0;
                }
            };
            streams(0, w);
            for (int q = 0; q < G; q++) {
                const int64_t i = (own + kCgOwners * (m + q)) * 32 + lane;
                const int rows = __shfl_sync(0xffffffffu, len, q);
                Rec6 o = {0, 0, 0, 0, 0, 0};
                if (i < n) o = load_rec(rec + i);
                double u0 = 0, u1 = 0, u2 = 0;
                for (int half = 0; half < 2; half++) {
                    double y0 = 0, y1 = 0, y2 = 0;
                    for (int k = w + 16 * half;;) {
                        Rec6 v[kCgRows];
                        double r[kCgRows];
#pragma unroll
                        for (int t = 0; t < kCgRows; t++) {
                            v[t] = load_rec(rec + j[t]);
                            r[t] = h[t];
                        }
                        k += 32 * kCgRows;
                        const bool more = k < rows;
                        if (more) streams(q, k);
                        else if (half == 0) streams(q, w + 16);
                        else if (q + 1 < G) streams(q + 1, w);
#pragma unroll
                        for (int t = 0; t < kCgRows; t++) {
                            const double c0 = v[t].x - o.x, c1 = v[t].y - o.y, c2 = v[t].z - o.z;
                            const double e = r[t] * (c0 * (o.px - v[t].px) + c1 * (o.py - v[t].py) + c2 * (o.pz - v[t].pz));
                            // a failed bond (scale 0) adds nothing, whatever its ends hold
                            y0 += r[t] != 0 ? e * c0 : 0.0;
                            y1 += r[t] != 0 ? e * c1 : 0.0;
                            y2 += r[t] != 0 ? e * c2 : 0.0;
                        }
                        if (!more) break;
                    }
                    u0 = half ? u0 + y0 : y0;
                    u1 = half ? u1 + y1 : y1;
                    u2 = half ? u2 + y2 : y2;
                }
                sm.acc[q][w][0][lane] = u0;
                sm.acc[q][w][1][lane] = u1;
                sm.acc[q][w][2][lane] = u2;
            }
            __syncthreads();
            for (int f = w; f < 3 * G; f += kCgWarps) {
                const int q = f / 3, c = f % 3;
                const int64_t i = (own + kCgOwners * (m + q)) * 32 + lane;
                double t[kCgWarps];
#pragma unroll
                for (int k = 0; k < kCgWarps; k++) t[k] = sm.acc[q][k][c][lane];
#pragma unroll
                for (int d = kCgWarps / 2; d > 0; d >>= 1)
#pragma unroll
                    for (int k = 0; k < d; k++) t[k] += t[k + d];
                if (i < n) {
                    const double v = g.held[i + c * n] ? 0.0 : t[0];
                    y[i + c * n] = v;
                    sm.py[q][c][lane] = (&rec[i].px)[c] * v;
                }
            }
            __syncthreads();
            if (w == 0)
                for (int q = 0; q < G; q++)
                    if ((own + kCgOwners * (m + q)) * 32 + lane < n)
                        for (int c = 0; c < 3; c++) acc += sm.py[q][c][lane];
        }
        if (w == 0) {
            double s = 0;
            for (int k = 0; k < 8; k++) s += __shfl_sync(0xffffffffu, acc, (lane & 3) * 8 + k);
            if (lane < 4) part[4 * own + lane] = make_double2(s, 0.0);
        }
    }
}

// The linear solve K delta = F on the free DOFs by conjugate gradients, one
// persistent launch: three barriers an iteration (after p.Kp, after r.z and
// r.r, after the new p) instead of six kernels, two of which summed 592 partials
// with one thread. In K p a lane stands for a node, so that a warp's 32
// neighbours lie side by side as the nodes do; a block shares out the partial sums
// of its slices, two per warp, so that warps and blocks are equally loaded at
// every size. Every sum keeps the order it had with a warp per node and a group
// of 8 warps per partial, so the iterates are those of the six kernels bit for
// bit: a different order moves a solution by the solve's tolerance, which flips last
// bits of positions and so changes single forces by 6e-8 of their RMS. What
// bounds it: at 20 000 nodes the latency of ten rounds of gathers, three barriers
// and the ordered sums of the partials, at millions the L1 wavefronts of the
// gathers and 12 bytes an entry. 20 000 nodes, 1.0M bonds, B200: 109 us an
// iteration with six kernels, 33 here.
// Warps with equal runs of rows and sums in any order took 22.
template <bool LISTS>
__global__ void __launch_bounds__(kCgThreads, 1) k_cg(CgArgs A)
{
    extern __shared__ __align__(16) unsigned char cg_smem[];
    CgShared &sm = *reinterpret_cast<CgShared *>(cg_smem);
    GridBarrier bar(A.bar, A.state + 2, A.timeout_ns);
    const int64_t n = A.g.n;
    const int groups = (int)min((int64_t)kCgGroups, (n + 255) / 256);
    const int pgroups = 4 * (int)min((int64_t)kCgOwners, A.g.ns);
    double2 *part0 = A.part, *part1 = A.part + kCgGroups;
    double rz, rr, rr0;
    int done = 0;
    if (A.first) {
        // delta = 0, r = F on the solved DOFs, z = M^-1 r, p = z
        node_sums(n, part0, sm, [&](int64_t i, double &rz_, double &rr_) {
            double ri[3], zi[3];
            for (int c = 0; c < 3; c++) ri[c] = A.skip[i + c * n] ? 0.0 : A.F[i + c * n];
            double m[6];
            for (int c = 0; c < 6; c++) m[c] = A.Minv[i + c * n];
            apply_minv(m, ri, zi);
            for (int c = 0; c < 3; c++) {
                if (A.skip[i + c * n]) zi[c] = 0.0;
                A.d[i + c * n] = 0.0;
                A.r[i + c * n] = ri[c];
                rz_ += ri[c] * zi[c];
                rr_ += ri[c] * ri[c];
            }
            A.rec[i].px = zi[0];
            A.rec[i].py = zi[1];
            A.rec[i].pz = zi[2];
        });
        if (!bar.wait()) return;
        const double2 s = add_groups(part0, groups, sm);
        rz = s.x;
        rr = rr0 = s.y;
    } else {
        rz = A.scal[0];
        rr = A.scal[1];
        rr0 = A.scal[2];
        done = A.state[1];
    }
    int state = rr0 > 0 ? CG_MORE : CG_DONE;   // a NaN r.r has nothing to solve either
    for (int it = 0; it < A.launch && state == CG_MORE; it++) {
        cg_product<LISTS>(A.g, A.rigE, A.rec, A.y, part1, sm);
        if (!bar.wait()) return;
        const double py = add_groups(part1, pgroups, sm).x;
        // delta += alpha p, r -= alpha y, z = M^-1 r
        const double alpha = py != 0 ? rz / py : 0.0;
        node_sums(n, part0, sm, [&](int64_t i, double &rz_, double &rr_) {
            // every load first: one round trip to L2
            const double pv[3] = {A.rec[i].px, A.rec[i].py, A.rec[i].pz};
            double ri[3], zi[3], di[3], m[6], yi[3];
            bool sk[3];
            for (int c = 0; c < 3; c++) {
                yi[c] = __ldcg(A.y + i + c * n);
                ri[c] = A.r[i + c * n];
                di[c] = A.d[i + c * n];
                sk[c] = A.skip[i + c * n] != 0;
            }
            for (int c = 0; c < 6; c++) m[c] = A.Minv[i + c * n];
            for (int c = 0; c < 3; c++) {
                A.d[i + c * n] = di[c] + alpha * pv[c];
                ri[c] = sk[c] ? 0.0 : ri[c] - alpha * yi[c];
                A.r[i + c * n] = ri[c];
            }
            apply_minv(m, ri, zi);
            for (int c = 0; c < 3; c++) {
                if (sk[c]) zi[c] = 0.0;
                A.z[i + c * n] = zi[c];
                rz_ += ri[c] * zi[c];
                rr_ += ri[c] * ri[c];
            }
        });
        if (!bar.wait()) return;
        const double2 s = add_groups(part0, groups, sm);
        // p = z + beta p
        const double beta = rz != 0 ? s.x / rz : 0.0;
        GRID_STRIDE(i, n)
        {
            A.rec[i].px = __ldcg(A.z + i) + beta * A.rec[i].px;
            A.rec[i].py = __ldcg(A.z + i + n) + beta * A.rec[i].py;
            A.rec[i].pz = __ldcg(A.z + i + 2 * n) + beta * A.rec[i].pz;
        }
        rz = s.x;
        rr = s.y;
        done++;
        if (done % kCgCheck == 0 || done == A.max_cg) {
            if (!isfinite(rr)) state = CG_NONFINITE;
            else if (rr <= A.tol2 * rr0 || done == A.max_cg) state = CG_DONE;
        }
        if (state == CG_MORE && !bar.wait()) return;
    }
    if (state == CG_DONE)
        GRID_STRIDE(i, n)
            for (int c = 0; c < 3; c++) A.x[i + c * n] += A.d[i + c * n];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        A.scal[0] = rz;
        A.scal[1] = rr;
        A.scal[2] = rr0;
        A.state[0] = state;
        A.state[1] = done;
    }
}

__global__ void k_prescribe(int64_t m, double *x, const uint8_t *__restrict__ held, double inc)
{
    GRID_STRIDE(e, m)
    if (held[e] == 2) x[e] += inc;
}

__global__ void k_iota(uint32_t *v, int64_t n) { GRID_STRIDE(i, n) v[i] = (uint32_t)i; }

__global__ void k_entry_keys(const uint32_t *__restrict__ a, const uint32_t *__restrict__ b, int64_t nB, uint32_t *key)
{
    GRID_STRIDE(q, 2 * nB) key[q] = (q & 1) ? b[q >> 1] : a[q >> 1];
}

__global__ void k_run_bounds(const uint32_t *__restrict__ skey, int64_t m, int64_t *first, int64_t *last)
{
    GRID_STRIDE(r, m)
    {
        const uint32_t p = skey[r];
        if (r == 0 || skey[r - 1] != p) first[p] = r;
        if (r == m - 1 || skey[r + 1] != p) last[p] = r + 1;
    }
}

__global__ void k_counts(const int64_t *__restrict__ first, const int64_t *__restrict__ last, int64_t n, int64_t *cnt)
{
    GRID_STRIDE(i, n + 1) cnt[i] = i < n ? last[i] - first[i] : 0;
}

}  // namespace

struct bbpd_static {
    int device = 0;
    cudaStream_t st = nullptr;
    int64_t n = 0, nB = 0;
    bbpd_params prm{};
    std::vector<void *> allocs;
    double *X = nullptr, *x = nullptr, *F = nullptr, *d = nullptr, *r = nullptr, *z = nullptr,
           *Minv = nullptr, *part = nullptr, *scal = nullptr, *red = nullptr, *rigE = nullptr;
    NodeRec *rec = nullptr;
    double2 *cg_part = nullptr;
    int *cg_state = nullptr;               // state, iterations, error word, barrier arrivals
    bool lists = false;                    // the solve's entries lie in lists, not in slices
    int64_t entries = 0;                   // of bond, col and rigE
    void (*cg)(CgArgs) = nullptr;
    int cg_grid = 0, cg_launch = kCgLaunch;
    unsigned long long cg_limit_ns = 0;    // of a barrier wait
    double *y = nullptr;
    uint8_t *skip = nullptr;
    SBonds b{};
    SNodes g{};
    template <class T>
    int alloc(T **q, size_t count)
    {
        BBPD_CUDA_TRY(cudaMalloc((void **)q, sizeof(T) * std::max<size_t>(count, 1)));
        allocs.push_back((void *)*q);
        return BBPD_OK;
    }
    ~bbpd_static()
    {
        if (st) cudaStreamSynchronize(st);
        for (void *q : allocs) cudaFree(q);
        if (st) cudaStreamDestroy(st);
    }
};

namespace {

// K delta = F on the free DOFs and x += delta; iterations and the outcome in
// state[0..1]. The host looks at the outcome once per launch.
int run_cg(bbpd_static *S, double cg_tol, int max_cg, int state[2])
{
    cudaStream_t st = S->st;
    CgArgs A{S->g, S->rigE, S->rec, S->F, S->Minv, S->skip, S->x, S->d, S->r, S->z, S->y, S->cg_part,
             S->scal, S->cg_state, reinterpret_cast<unsigned *>(S->cg_state + 3), S->cg_limit_ns,
             cg_tol * cg_tol, 1, max_cg, S->cg_launch};
    for (;; A.first = 0) {
        BBPD_CUDA_TRY(cudaMemsetAsync(S->cg_state + 2, 0, 2 * sizeof(int), st));
        void *args[] = {(void *)&A};
        BBPD_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)S->cg, dim3(S->cg_grid), dim3(kCgThreads), args, sizeof(CgShared), st));
        int h[3];
        BBPD_CUDA_TRY(cudaMemcpyAsync(h, S->cg_state, sizeof(h), cudaMemcpyDeviceToHost, st));
        BBPD_CUDA_TRY(cudaStreamSynchronize(st));
        if (h[2] & ERR_TIMEOUT) return fail(BBPD_ERR_TIMEOUT, "grid barrier wait exceeded its limit; kernel returned early");
        state[0] = h[0];
        state[1] = h[1];
        if (h[0] != CG_MORE) return BBPD_OK;
    }
}

int read_scalars(bbpd_static *S, const double *src, int cnt, double *out)
{
    BBPD_CUDA_TRY(cudaMemcpyAsync(out, src, sizeof(double) * cnt, cudaMemcpyDeviceToHost, S->st));
    BBPD_CUDA_TRY(cudaStreamSynchronize(S->st));
    return BBPD_OK;
}

}  // namespace

extern "C" int bbpd_static_create(const bbpd_problem *pb, const bbpd_params *prm, int device, bbpd_static **out)
{
    clear_error();
    if (!pb || !prm || !out) return fail(BBPD_ERR_ARG, "null argument");
    *out = nullptr;
    TRY(require_device());
    const int64_t n = pb->n_nodes, nB = pb->n_bonds;
    if (n < 1 || n >= ((int64_t)1 << 31) || nB < 0 || nB >= ((int64_t)1 << 31))
        return fail(BBPD_ERR_ARG, "need 1 <= n_nodes < 2^31 and 0 <= n_bonds < 2^31");
    if (!pb->undeformed_coordinates || (nB && (!pb->bondlist || !pb->undeformed_length || !pb->bond_stiffness ||
                                               !pb->volume_correction)))
        return fail(BBPD_ERR_ARG, "missing coordinates or bond arrays");
    if (prm->law < 0 || prm->law > 3) return fail(BBPD_ERR_ARG, "bad law");
    if (!(prm->failure_functionality == 0.0 || prm->failure_functionality == 1.0))
        return fail(BBPD_ERR_UNSUPPORTED, "failure_functionality must be 0 or 1");
    if (pb->s0 || pb->s1 || pb->sc) return fail(BBPD_ERR_UNSUPPORTED, "the static solver takes scalar law stretches");
    const double *bl = pb->bondlist;
    std::vector<uint32_t> a(nB), bb(nB);
    std::vector<uint8_t> bt(nB, 0);
    std::vector<double> bfm(nB, 1.0), fl(nB, 1.0);
    for (int64_t k = 0; k < nB; k++) {
        const double ai = bl[k], bj = bl[nB + k];
        if (!(ai >= 1 && bj >= 1 && ai <= (double)n && bj <= (double)n && ai == std::floor(ai) && bj == std::floor(bj)))
            return fail(BBPD_ERR_ARG, "BONDLIST row %lld is not a pair of node ids", (long long)k + 1);
        a[k] = (uint32_t)(ai - 1);
        bb[k] = (uint32_t)(bj - 1);
        if (pb->bond_type) {
            const double t = pb->bond_type[k];
            if (!(t == 0 || t == 1 || t == 2)) return fail(BBPD_ERR_ARG, "BONDTYPE[%lld] = %g", (long long)k, t);
            bt[k] = (uint8_t)t;
            bfm[k] = t == 1 ? 3.0 : 1.0;   // buildbonddata.m:70-71
        }
        if (pb->fail) {
            const double f = pb->fail[k];
            if (!(f == 0 || f == 1)) return fail(BBPD_ERR_ARG, "fail[%lld] = %g", (long long)k, f);
            fl[k] = f;
        }
        if (pb->stretch_plastic && pb->stretch_plastic[k] != 0)
            return fail(BBPD_ERR_UNSUPPORTED, "non-zero stretchPlastic is not on this path");
    }
    std::vector<uint8_t> held(3 * n, 0);
    for (int64_t e = 0; e < 3 * n; e++) {
        const bool cf = pb->constraint_flag && pb->constraint_flag[e] == 1;
        const bool pf = pb->prescribed_flag && pb->prescribed_flag[e] == 1;
        held[e] = cf ? 1 : (pf ? 2 : 0);   // a support holds a DOF even where a load is prescribed
    }
    if (cudaSetDevice(device) != cudaSuccess) {
        cudaGetLastError();
        return fail(BBPD_ERR_CUDA, "cudaSetDevice(%d) failed", device);
    }
    auto *S = new bbpd_static;
    std::unique_ptr<bbpd_static> guard(S);
    S->device = device;
    S->n = n;
    S->nB = nB;
    S->prm = *prm;
    BBPD_CUDA_TRY(cudaStreamCreateWithFlags(&S->st, cudaStreamNonBlocking));
    cudaStream_t st = S->st;
    TRY(S->alloc(&S->X, 3 * n));
    TRY(S->alloc(&S->x, 3 * n));
    TRY(staging::upload_copy(S->X, pb->undeformed_coordinates, 3 * n, st));
    BBPD_CUDA_TRY(cudaMemcpyAsync(S->x, S->X, sizeof(double) * 3 * n, cudaMemcpyDeviceToDevice, st));
    for (double **q : {&S->F, &S->d, &S->r, &S->z}) TRY(S->alloc(q, 3 * n));
    TRY(S->alloc(&S->rec, n));
    TRY(S->alloc(&S->Minv, 6 * n));
    TRY(S->alloc(&S->skip, 3 * n));
    TRY(S->alloc(&S->part, 2 * kRedBlocks));
    TRY(S->alloc(&S->scal, 4));
    TRY(S->alloc(&S->red, 2));
    BBPD_CUDA_TRY(cudaMemsetAsync(S->F, 0, sizeof(double) * 3 * n, st));

    SBonds &B = S->b;
    uint32_t *da = nullptr, *db = nullptr;
    uint8_t *dbt = nullptr, *dheld = nullptr;
    double *dL0 = nullptr, *dBS = nullptr, *dV = nullptr, *dBFM = nullptr;
    TRY(S->alloc(&da, nB));
    TRY(S->alloc(&db, nB));
    TRY(S->alloc(&dbt, nB));
    TRY(S->alloc(&dL0, nB));
    TRY(S->alloc(&dBS, nB));
    TRY(S->alloc(&dV, nB));
    TRY(S->alloc(&dBFM, nB));
    TRY(S->alloc(&B.fail, nB));
    TRY(S->alloc(&B.bsf, nB));
    TRY(S->alloc(&B.flag, nB));
    TRY(S->alloc(&B.rig, nB));
    TRY(S->alloc(&B.f, 3 * nB));
    TRY(S->alloc(&dheld, 3 * n));
    TRY(staging::upload_copy(da, a.data(), nB, st));
    TRY(staging::upload_copy(db, bb.data(), nB, st));
    TRY(staging::upload_copy(dbt, bt.data(), nB, st));
    TRY(staging::upload_copy(dBFM, bfm.data(), nB, st));
    TRY(staging::upload_copy(B.fail, fl.data(), nB, st));
    TRY(staging::upload_copy(dheld, held.data(), 3 * n, st));
    if (nB) {
        TRY(staging::upload_copy(dL0, pb->undeformed_length, nB, st));
        TRY(staging::upload_copy(dBS, pb->bond_stiffness, nB, st));
        TRY(staging::upload_copy(dV, pb->volume_correction, nB, st));
    }
    BBPD_CUDA_TRY(cudaMemsetAsync(B.bsf, 0, sizeof(double) * std::max<int64_t>(nB, 1), st));
    BBPD_CUDA_TRY(cudaMemsetAsync(B.flag, 0, std::max<int64_t>(nB, 1), st));
    B.a = da;
    B.b = db;
    B.L0 = dL0;
    B.BS = dBS;
    B.VCF = dV;
    B.BFM = dBFM;
    B.BT = dbt;
    B.nB = nB;
    B.law = prm->law;
    B.V = prm->cell_volume;
    LawScalars &P = B.P;
    P.s0 = prm->s0;
    P.s1 = prm->s1;
    P.sc = prm->sc;
    P.beta = prm->beta_tri;
    const double eta = prm->s1 / prm->s0;
    P.tri_c1 = (eta - P.beta) / (eta - 1);
    P.tri_c2 = (1 - P.beta) / (eta - 1);
    P.k = prm->k_exp;
    P.alpha = prm->alpha_exp;
    P.exp_den = 1 - std::exp(-prm->k_exp);
    P.sc_steel = prm->sc_steel;
    P.ff = prm->failure_functionality;

    // per-node lists of bond ends in bond order: stable sort of q = 2k + side by node
    const int64_t m = 2 * nB;   // list entries
    int64_t *off = nullptr;
    uint32_t *ent = nullptr;
    TRY(S->alloc(&off, n + 1));
    TRY(S->alloc(&ent, m));
    {
        uint32_t *key = nullptr, *skey = nullptr, *val = nullptr;
        int64_t *first = nullptr, *last = nullptr, *cnt = nullptr;
        uint8_t *tmp = nullptr;
        size_t tb = 0, ts = 0;
        int bits = 1;
        while (bits < 32 && ((int64_t)1 << bits) < n) bits++;
        BBPD_CUDA_TRY(cudaMallocAsync(&key, sizeof(uint32_t) * std::max<int64_t>(m, 1), st));
        BBPD_CUDA_TRY(cudaMallocAsync(&skey, sizeof(uint32_t) * std::max<int64_t>(m, 1), st));
        BBPD_CUDA_TRY(cudaMallocAsync(&val, sizeof(uint32_t) * std::max<int64_t>(m, 1), st));
        BBPD_CUDA_TRY(cudaMallocAsync(&first, sizeof(int64_t) * n, st));
        BBPD_CUDA_TRY(cudaMallocAsync(&last, sizeof(int64_t) * n, st));
        BBPD_CUDA_TRY(cudaMallocAsync(&cnt, sizeof(int64_t) * (n + 1), st));
        BBPD_CUDA_TRY(cudaMemsetAsync(first, 0, sizeof(int64_t) * n, st));
        BBPD_CUDA_TRY(cudaMemsetAsync(last, 0, sizeof(int64_t) * n, st));
        if (m > 0) {
            k_entry_keys<<<blocks_for(m), kThreads, 0, st>>>(da, db, nB, key);
            k_iota<<<blocks_for(m), kThreads, 0, st>>>(val, m);
            BBPD_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tb, key, skey, val, ent, m, 0, bits, st));
        }
        BBPD_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, ts, cnt, off, n + 1, st));
        BBPD_CUDA_TRY(cudaMallocAsync(&tmp, std::max<size_t>(std::max(tb, ts), 1), st));
        int rc = BBPD_OK;
        if (m > 0) {
            cudaError_t e = cub::DeviceRadixSort::SortPairs(tmp, tb, key, skey, val, ent, m, 0, bits, st);
            if (e == cudaSuccess) {
                k_run_bounds<<<blocks_for(m), kThreads, 0, st>>>(skey, m, first, last);
                e = cudaGetLastError();
            }
            if (e != cudaSuccess) rc = fail(BBPD_ERR_CUDA, "static solver lists: %s", cudaGetErrorString(e));
        }
        if (rc == BBPD_OK) {
            k_counts<<<blocks_for(n + 1), kThreads, 0, st>>>(first, last, n, cnt);
            size_t t2 = std::max(tb, ts);
            cudaError_t e = cub::DeviceScan::ExclusiveSum(tmp, t2, cnt, off, n + 1, st);
            if (e != cudaSuccess) rc = fail(BBPD_ERR_CUDA, "static solver lists: %s", cudaGetErrorString(e));
        }
        for (void *q : {(void *)key, (void *)skey, (void *)val, (void *)first, (void *)last, (void *)cnt, (void *)tmp})
            cudaFreeAsync(q, st);
        TRY(rc);
    }
    // the same lists in slices of 32 nodes
    const int64_t ns = (n + 31) / 32;
    int64_t *sptr = nullptr, slots = 0;
    uint32_t *bond = nullptr, *col = nullptr;
    TRY(S->alloc(&sptr, ns + 1));
    {
        int64_t *cnt = nullptr;
        uint8_t *tmp = nullptr;
        size_t tb = 0;
        BBPD_CUDA_TRY(cudaMallocAsync(&cnt, sizeof(int64_t) * (ns + 1), st));
        k_slice_lengths<<<blocks_for(32 * (ns + 1)), kThreads, 0, st>>>(off, n, ns, cnt);
        cudaError_t e = cub::DeviceScan::ExclusiveSum(nullptr, tb, cnt, sptr, ns + 1, st);
        if (e == cudaSuccess) e = cudaMallocAsync(&tmp, std::max<size_t>(tb, 1), st);
        if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(tmp, tb, cnt, sptr, ns + 1, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&slots, sptr + ns, sizeof(int64_t), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        cudaFreeAsync(cnt, st);
        if (tmp) cudaFreeAsync(tmp, st);
        if (e != cudaSuccess) return fail(BBPD_ERR_CUDA, "static solver slices: %s", cudaGetErrorString(e));
    }
    // Slices where padding takes at most three quarters of them (a beam's take under
    // 1.3 times its entries): 16 bytes a slot, read a row at a time. Beyond, the memory
    // would be the longest lists' 32-fold: 20 000 nodes, 64 of them bonded to all
    // others, took 910 MB against 306 with lists, and 400 iterations 275 ms against
    // 172 (552 with six kernels an iteration).
    S->lists = slots > 4 * m;
    S->entries = S->lists ? m : slots;
    // one allocation for the three arrays: mapping and unmapping one takes 0.4 ms
    TRY(S->alloc(&S->rigE, 2 * S->entries));
    bond = reinterpret_cast<uint32_t *>(S->rigE + S->entries);
    col = bond + S->entries;
    if (S->lists) k_list_fill<<<blocks_for(m), kThreads, 0, st>>>(ent, da, db, m, bond, col);
    else k_slice_fill<<<blocks_for(32 * ns), kThreads, 0, st>>>(off, ent, da, db, n, ns, sptr, bond, col);
    TRY(launch_check());
    int nsm = 0, occ = 0, coop = 0;
    BBPD_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device));
    BBPD_CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device));
    if (!coop) return fail(BBPD_ERR_UNSUPPORTED, "device lacks cooperative launch");
    S->cg = S->lists ? k_cg<true> : k_cg<false>;
    BBPD_CUDA_TRY(cudaFuncSetAttribute(S->cg, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(CgShared)));
    BBPD_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, S->cg, kCgThreads, sizeof(CgShared)));
    if (occ < 1) return fail(BBPD_ERR_CUDA, "kernel cannot be resident");
    // a block for every owner with slices
    S->cg_grid = (int)std::max<int64_t>(1, std::min<int64_t>({(int64_t)nsm, (int64_t)kCgOwners, ns}));
    // A solve that makes progress never waits this long: 10 s, and 0.1 us for every
    // row of 32 entries, should one block have them all (16 warps take one in 0.02 us).
    // barrier_timeout_s, the limit of the time-stepping kernels, may be short; it
    // has no say here.
    S->cg_limit_ns = 10000000000ull + 100ull * (unsigned long long)(slots >> 5);
    TRY(S->alloc(&S->y, 3 * n));
    TRY(S->alloc(&S->cg_part, 2 * kCgGroups));
    TRY(S->alloc(&S->cg_state, 4));
    S->g.off = off;
    S->g.ent = ent;
    S->g.sptr = sptr;
    S->g.bond = bond;
    S->g.col = col;
    S->g.ns = ns;
    S->g.held = dheld;
    S->g.n = n;
    S->g.nB = nB;
    BBPD_CUDA_TRY(cudaStreamSynchronize(st));
    *out = guard.release();
    return BBPD_OK;
}

extern "C" int bbpd_static_step(bbpd_static *S, double increment, double tol, int max_newton, double cg_tol,
                                int max_cg, bbpd_static_stats *stats)
{
    if (!S || !stats) return fail(BBPD_ERR_ARG, "null argument");
    if (!(tol > 0) || !(cg_tol > 0) || max_newton < 1 || max_cg < 1 || !std::isfinite(increment))
        return fail(BBPD_ERR_ARG, "need tol > 0, cg_tol > 0, max_newton >= 1, max_cg >= 1, finite increment");
    BBPD_CUDA_TRY(cudaSetDevice(S->device));
    cudaStream_t st = S->st;
    const int64_t n = S->n;
    *stats = bbpd_static_stats{};
    if (increment != 0) k_prescribe<<<blocks_for(3 * n), kThreads, 0, st>>>(3 * n, S->x, S->g.held, increment);
    for (int it = 0;; it++) {
        k_static_bonds<<<blocks_for(S->nB), kThreads, 0, st>>>(S->b, S->x, n);
        k_static_nodal<<<kRedBlocks, kThreads, 0, st>>>(S->g, S->b.f, S->prm.cell_volume, S->F, S->part);
        k_reduce<<<1, 64, 0, st>>>(S->part, kRedBlocks, 2, S->red);
        TRY(launch_check());
        double rr[2];
        TRY(read_scalars(S, S->red, 2, rr));
        stats->residual = std::sqrt(rr[0]);
        stats->reaction = std::sqrt(rr[1]);
        stats->newton_iterations = it;
        if (!std::isfinite(stats->residual) || !std::isfinite(stats->reaction))
            return fail(BBPD_ERR_NONFINITE, "non-finite nodal force");
        if (stats->residual <= tol * stats->reaction || stats->residual == 0) {
            stats->converged = 1;
            return BBPD_OK;
        }
        if (it == max_newton) return BBPD_OK;   // not converged: stats say so
        // K delta = F on the free DOFs by PCG, x += delta
        k_static_records<<<blocks_for(n), kThreads, 0, st>>>(S->x, n, S->rec);
        k_slot_rig<<<blocks_for(S->entries), kThreads, 0, st>>>(S->g.bond, S->b.rig, S->entries, S->rigE);
        (S->lists ? k_static_precond<true> : k_static_precond<false>)<<<blocks_for(n), kThreads, 0, st>>>(
            S->g, S->rigE, S->rec, S->Minv, S->skip);
        TRY(launch_check());
        int cg[2] = {CG_DONE, 0};
        TRY(run_cg(S, cg_tol, max_cg, cg));
        stats->cg_iterations += cg[1];
        if (cg[0] == CG_NONFINITE) return fail(BBPD_ERR_NONFINITE, "conjugate gradient diverged");
    }
}

extern "C" int bbpd_selftest_static_launch(bbpd_static *S, int iterations, double limit_s)
{
    if (!S || iterations < 1 || !(limit_s >= 0) || limit_s > 1e6)
        return fail(BBPD_ERR_ARG, "need a solver, iterations >= 1 and 0 <= limit_s <= 1e6");
    S->cg_launch = iterations;
    if (limit_s > 0) S->cg_limit_ns = (unsigned long long)(limit_s * 1e9);
    return BBPD_OK;
}

extern "C" int bbpd_static_get(bbpd_static *S, int field, double *out)
{
    if (!S || !out) return fail(BBPD_ERR_ARG, "null argument");
    BBPD_CUDA_TRY(cudaSetDevice(S->device));
    cudaStream_t st = S->st;
    const int64_t n = S->n, nB = S->nB;
    switch (field) {
    case BBPD_FIELD_DEFORMED: return staging::download_copy(out, S->x, 3 * n, st);
    case BBPD_FIELD_FORCE: return staging::download_copy(out, S->F, 3 * n, st);
    case BBPD_FIELD_DISPLACEMENT: {
        const double *x = S->x;
        TRY(staging::download_copy(out, x, 3 * n, st));
        std::vector<double> X(3 * n);
        TRY(staging::download_copy(X.data(), S->X, 3 * n, st));
        for (int64_t e = 0; e < 3 * n; e++) out[e] = out[e] - X[e];
        return BBPD_OK;
    }
    case BBPD_FIELD_BSF: return staging::download_copy(out, S->b.bsf, nB, st);
    case BBPD_FIELD_FAIL: return staging::download_copy(out, S->b.fail, nB, st);
    case BBPD_FIELD_FLAG: {
        std::vector<uint8_t> f(nB);
        TRY(staging::download_copy(f.data(), S->b.flag, nB, st));
        for (int64_t k = 0; k < nB; k++) out[k] = f[k];
        return BBPD_OK;
    }
    default: return fail(BBPD_ERR_ARG, "field %d not held by the static solver", field);
    }
}

extern "C" int bbpd_static_destroy(bbpd_static *S)
{
    if (!S) return BBPD_OK;
    cudaSetDevice(S->device);
    delete S;
    return BBPD_OK;
}

// ---- buildstiffnessmatrixCSCformat.m as a routine ----

namespace {

struct CooBonds {
    const double *X;            // nodal coordinates, nNodes x NOD
    const double *bl, *VCF, *BS, *BFM, *fail, *BSF;
    int64_t n, nB;
    int NOD;
    double V;
};

// Local stiffness of bond k: its scale rig and bond vector (NOD components);
// false for a failed bond (buildstiffnessmatrixCSCformat.m:72, :110).
__device__ __forceinline__ bool coo_local(const CooBonds &q, int64_t k, double &rig, double c[3], int64_t &i,
                                          int64_t &j)
{
    if (q.fail[k] != 1) return false;
    i = (int64_t)q.bl[k] - 1;
    j = (int64_t)q.bl[q.nB + k] - 1;
    double L2 = 0;
    for (int u = 0; u < q.NOD; u++) {
        c[u] = q.X[j + u * q.n] - q.X[i + u * q.n];
        L2 = u == 0 ? c[u] * c[u] : L2 + c[u] * c[u];
    }
    const double L = sqrt(L2);
    if (q.NOD == 3)   // :116
        rig = q.BFM[k] * ((q.BS[k] / (L * L * L)) * q.VCF[k] * (q.V * q.V)) * (1 - q.BSF[k]);
    else              // :78
        rig = q.BFM[k] * (q.BS[k] / (L * L * L)) * q.VCF[k] * (q.V * q.V);
    return true;
}

// entry (r, s) of the 2 NOD x 2 NOD local matrix rig [A -A; -A A], A = c c^T
__device__ __forceinline__ double coo_entry(double rig, const double *c, int NOD, int r, int s)
{
    const double m = c[r % NOD] * c[s % NOD];
    return ((r < NOD) == (s < NOD)) ? rig * m : rig * (-m);
}

// nonzero count and norm(Klocal) of every bond; norm = 2 |rig| |c|^2, the
// largest singular value of rig [A -A; -A A]
__global__ void k_coo_count(CooBonds q, int64_t *cnt, double *nrm)
{
    GRID_STRIDE(k, q.nB + 1)
    {
        if (k == q.nB) {
            cnt[k] = 0;
            continue;
        }
        double rig, c[3];
        int64_t i, j;
        int64_t z = 0;
        double nm = 0;
        if (coo_local(q, k, rig, c, i, j)) {
            const int D = 2 * q.NOD;
            for (int s = 0; s < D; s++)
                for (int r = 0; r < D; r++) z += coo_entry(rig, c, q.NOD, r, s) != 0;
            double L2 = 0;
            for (int u = 0; u < q.NOD; u++) L2 = u == 0 ? c[u] * c[u] : L2 + c[u] * c[u];
            nm = 2 * fabs(rig) * L2;
        }
        cnt[k] = z;
        nrm[k] = nm;
    }
}

// nonzeros of every bond in MATLAB find order (column-major), with 1-based
// global DOFs NOD (node - 1) + 1 .. NOD node (:91-100, :129-138)
__global__ void k_coo_write(CooBonds q, const int64_t *__restrict__ off, double *rows, double *cols, double *vals)
{
    GRID_STRIDE(k, q.nB)
    {
        double rig, c[3];
        int64_t i, j;
        if (!coo_local(q, k, rig, c, i, j)) continue;
        const int D = 2 * q.NOD;
        int64_t o = off[k];
        for (int s = 0; s < D; s++)
            for (int r = 0; r < D; r++) {
                const double v = coo_entry(rig, c, q.NOD, r, s);
                if (v == 0) continue;
                const int64_t gr = (r < q.NOD ? q.NOD * i : q.NOD * j) + (r % q.NOD) + 1;
                const int64_t gc = (s < q.NOD ? q.NOD * i : q.NOD * j) + (s % q.NOD) + 1;
                rows[o] = (double)gr;
                cols[o] = (double)gc;
                vals[o] = v;
                o++;
            }
    }
}

__global__ void k_node_sum(const int64_t *__restrict__ off, const uint32_t *__restrict__ ent, int64_t n,
                           const double *__restrict__ v, double *out)
{
    GRID_STRIDE(i, n)
    {
        double a = 0;
        for (int64_t e = off[i]; e < off[i + 1]; e++) a = a + v[ent[e] >> 1];
        out[i] = a;
    }
}

__global__ void k_bl_nodes(const double *__restrict__ bl, int64_t nB, int64_t n, uint32_t *a, uint32_t *b, int *bad)
{
    GRID_STRIDE(k, nB)
    {
        const double x = bl[k], y = bl[nB + k];
        if (!(x >= 1 && y >= 1 && x <= (double)n && y <= (double)n)) {
            *bad = 1;
            a[k] = b[k] = 0;
            continue;
        }
        a[k] = (uint32_t)(x - 1);
        b[k] = (uint32_t)(y - 1);
    }
}

}  // namespace

extern "C" int bbpd_dev_buildstiffnessmatrix(const double *X, int64_t nNodes, int NOD, const double *BONDLIST,
        const double *VCF, double VOLUME, const double *BS, const double *BFM, const double *failFlag, const double *BSF,
        int64_t nBonds, int64_t capacity, int64_t *nnz, double *rowIndex, double *columnIndex, double *values,
        double *massVector, void *stream)
{
    if (!nnz) return fail(BBPD_ERR_ARG, "null nnz");
    if (NOD != 2 && NOD != 3) return fail(BBPD_ERR_ARG, "NOD must be 2 or 3");
    if (nNodes < 1 || nNodes >= ((int64_t)1 << 31) || nBonds < 0 || nBonds >= ((int64_t)1 << 31))
        return fail(BBPD_ERR_ARG, "need 1 <= nNodes < 2^31 and 0 <= nBonds < 2^31");
    if (!X || (nBonds && (!BONDLIST || !VCF || !BS || !BFM || !failFlag || !BSF))) return fail(BBPD_ERR_ARG, "null array");
    TRY(require_device());
    cudaStream_t st = as_stream(stream);
    const int64_t n = nNodes, nB = nBonds, m = 2 * nB;
    CooBonds q{X, BONDLIST, VCF, BS, BFM, failFlag, BSF, n, nB, NOD, VOLUME};
    std::vector<void *> tmp;
    auto get = [&](void **p, size_t bytes) -> int {
        BBPD_CUDA_TRY(scratch_malloc(p, std::max<size_t>(bytes, 8), st));
        tmp.push_back(*p);
        return BBPD_OK;
    };
    struct Free {
        std::vector<void *> &t;
        cudaStream_t s;
        ~Free()
        {
            for (void *p : t) cudaFreeAsync(p, s);
        }
    } freer{tmp, st};
    uint32_t *a = nullptr, *b = nullptr, *key = nullptr, *skey = nullptr, *val = nullptr, *ent = nullptr;
    int64_t *cnt = nullptr, *off = nullptr, *first = nullptr, *last = nullptr, *ncnt = nullptr, *noff = nullptr;
    double *nrm = nullptr;
    int *bad = nullptr;
    TRY(get((void **)&a, 4 * nB));
    TRY(get((void **)&b, 4 * nB));
    TRY(get((void **)&bad, sizeof(int)));
    TRY(get((void **)&cnt, 8 * (nB + 1)));
    TRY(get((void **)&off, 8 * (nB + 1)));
    TRY(get((void **)&nrm, 8 * nB));
    BBPD_CUDA_TRY(cudaMemsetAsync(bad, 0, sizeof(int), st));
    k_bl_nodes<<<blocks_for(nB), kThreads, 0, st>>>(BONDLIST, nB, n, a, b, bad);
    k_coo_count<<<blocks_for(nB + 1), kThreads, 0, st>>>(q, cnt, nrm);
    TRY(launch_check());
    size_t tb = 0;
    BBPD_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tb, cnt, off, nB + 1, st));
    void *t1 = nullptr;
    TRY(get(&t1, tb));
    BBPD_CUDA_TRY(cub::DeviceScan::ExclusiveSum(t1, tb, cnt, off, nB + 1, st));
    int64_t total = 0;
    int hbad = 0;
    BBPD_CUDA_TRY(cudaMemcpyAsync(&total, off + nB, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    BBPD_CUDA_TRY(cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, st));
    BBPD_CUDA_TRY(cudaStreamSynchronize(st));
    if (hbad) return fail(BBPD_ERR_ARG, "BONDLIST holds node ids outside [1, nNodes]");
    *nnz = total;
    if (capacity >= total && total > 0 && rowIndex && columnIndex && values) {
        k_coo_write<<<blocks_for(nB), kThreads, 0, st>>>(q, off, rowIndex, columnIndex, values);
        TRY(launch_check());
    }
    if (massVector) {
        // massVector(i) accumulates norm(Klocal) of its intact bonds in bond order
        TRY(get((void **)&key, 4 * m));
        TRY(get((void **)&skey, 4 * m));
        TRY(get((void **)&val, 4 * m));
        TRY(get((void **)&ent, 4 * m));
        TRY(get((void **)&first, 8 * n));
        TRY(get((void **)&last, 8 * n));
        TRY(get((void **)&ncnt, 8 * (n + 1)));
        TRY(get((void **)&noff, 8 * (n + 1)));
        BBPD_CUDA_TRY(cudaMemsetAsync(first, 0, 8 * n, st));
        BBPD_CUDA_TRY(cudaMemsetAsync(last, 0, 8 * n, st));
        int bits = 1;
        while (bits < 32 && ((int64_t)1 << bits) < n) bits++;
        if (m > 0) {
            k_entry_keys<<<blocks_for(m), kThreads, 0, st>>>(a, b, nB, key);
            k_iota<<<blocks_for(m), kThreads, 0, st>>>(val, m);
            BBPD_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tb, key, skey, val, ent, m, 0, bits, st));
            void *t2 = nullptr;
            TRY(get(&t2, tb));
            BBPD_CUDA_TRY(cub::DeviceRadixSort::SortPairs(t2, tb, key, skey, val, ent, m, 0, bits, st));
            k_run_bounds<<<blocks_for(m), kThreads, 0, st>>>(skey, m, first, last);
        }
        k_counts<<<blocks_for(n + 1), kThreads, 0, st>>>(first, last, n, ncnt);
        BBPD_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tb, ncnt, noff, n + 1, st));
        void *t3 = nullptr;
        TRY(get(&t3, tb));
        BBPD_CUDA_TRY(cub::DeviceScan::ExclusiveSum(t3, tb, ncnt, noff, n + 1, st));
        k_node_sum<<<blocks_for(n), kThreads, 0, st>>>(noff, ent, n, nrm, massVector);
        TRY(launch_check());
    }
    BBPD_CUDA_TRY(cudaStreamSynchronize(st));
    return BBPD_OK;
}

extern "C" int bbpd_buildstiffnessmatrix(const double *X, int64_t nNodes, int NOD, const double *BONDLIST,
        const double *VCF, double VOLUME, const double *BS, const double *BFM, const double *failFlag, const double *BSF,
        int64_t nBonds, int64_t capacity, int64_t *nnz, double *rowIndex, double *columnIndex, double *values,
        double *massVector)
{
    if (!nnz) return fail(BBPD_ERR_ARG, "null nnz");
    if (NOD != 2 && NOD != 3) return fail(BBPD_ERR_ARG, "NOD must be 2 or 3");
    if (nNodes < 1 || nBonds < 0) return fail(BBPD_ERR_ARG, "bad sizes");
    if (!X || (nBonds && (!BONDLIST || !VCF || !BS || !BFM || !failFlag || !BSF))) return fail(BBPD_ERR_ARG, "null array");
    TRY(require_device());
    cudaStream_t st = nullptr;
    BBPD_CUDA_TRY(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    struct Own {
        cudaStream_t s;
        std::vector<void *> p;
        ~Own()
        {
            for (void *q : p) cudaFreeAsync(q, s);
            cudaStreamSynchronize(s);
            cudaStreamDestroy(s);
        }
    } own{st, {}};
    auto up = [&](const double *h, int64_t cnt, double **d) -> int {
        BBPD_CUDA_TRY(scratch_malloc((void **)d, sizeof(double) * std::max<int64_t>(cnt, 1), st));
        own.p.push_back(*d);
        return h ? staging::upload_copy(*d, h, cnt, st) : BBPD_OK;
    };
    const int64_t nB = nBonds;
    double *dX, *dbl, *dV, *dBS, *dBFM, *dfail, *dBSF, *dm = nullptr;
    TRY(up(X, NOD * nNodes, &dX));
    TRY(up(BONDLIST, 2 * nB, &dbl));
    TRY(up(VCF, nB, &dV));
    TRY(up(BS, nB, &dBS));
    TRY(up(BFM, nB, &dBFM));
    TRY(up(failFlag, nB, &dfail));
    TRY(up(BSF, nB, &dBSF));
    if (massVector) TRY(up(nullptr, nNodes, &dm));
    TRY(bbpd_dev_buildstiffnessmatrix(dX, nNodes, NOD, dbl, dV, VOLUME, dBS, dBFM, dfail, dBSF, nB, 0, nnz, nullptr,
                                      nullptr, nullptr, dm, st));
    const int64_t total = *nnz;
    if (capacity >= total && total > 0 && rowIndex && columnIndex && values) {
        double *dr, *dc, *dv;
        TRY(up(nullptr, total, &dr));
        TRY(up(nullptr, total, &dc));
        TRY(up(nullptr, total, &dv));
        int64_t again = 0;
        TRY(bbpd_dev_buildstiffnessmatrix(dX, nNodes, NOD, dbl, dV, VOLUME, dBS, dBFM, dfail, dBSF, nB, total, &again,
                                          dr, dc, dv, nullptr, st));
        TRY(staging::download_copy(rowIndex, dr, total, st));
        TRY(staging::download_copy(columnIndex, dc, total, st));
        TRY(staging::download_copy(values, dv, total, st));
    }
    if (dm) TRY(staging::download_copy(massVector, dm, nNodes, st));
    return BBPD_OK;
}
