// Persistent PCG for scenes whose rows are few enough that a CTA can keep its share on chip:
// the matrix rows in shared memory and the CG vectors in registers, for the whole solve.  Several scenes
// run as independent teams of CTAs in one launch, each with its own barrier and its own end.
//
// The streaming kernel (fem_pcg.cu) reads the matrix from L2 or DRAM every iteration and meets two
// grid barriers; below about 100,000 nodes neither the bytes nor the operations bound it but the
// chain of dependent latencies (13-17 us per iteration from 5,000 to 50,000 nodes, of which the
// bytes need 1-4).  Here
//   * a CTA copies its rows' blocks to shared memory once per launch (a uniform share of every row's
//     columns when they do not all fit; the rest is read from L2 each iteration);
//   * the columns its rows touch are listed once (own rows, then the halo), with a 16-bit local
//     column per stored block.  An iteration computes the search direction once per listed column
//     into shared memory, and the product reads nothing else;
//   * the columns of a slice are dealt to several warps, whose partial sums are added in a fixed
//     order, so a row's product is a chain of a few loads instead of its whole length;
//   * one reduction per iteration instead of two where several CTAs meet (a CTA that is alone keeps both, as
//     CTA barriers).
//
// One reduction (predict and recompute: Meurant 1987; Chen and Carson, "Predict-and-recompute
// conjugate gradient variants", 2020).  With s = A p and t = M s, one pass forms
//   p.s, z.s, t.s, r.z, r.r, r.s, s.s
// so alpha = r.z / p.s, and the next iteration's scalars are predicted before r is updated:
//   (r.z)' = r.z - 2 alpha z.s + alpha^2 t.s,   (r.r)' = r.r - 2 alpha r.s + alpha^2 s.s.
// beta and the stopping test use the predictions, alpha the recomputed r.z, and z = M r is formed
// from the updated r each time, so the iterates are standard CG's up to rounding.  A prediction that
// cancels (a drop below kPredictFloor of the old value) is replaced by the sums themselves, in a
// second reduction.  A neighbour's next direction p' = (z - alpha t) + beta p follows from its
// 48-byte record (z, p, t), published before the reduction, by the owner's own expression.
//
// Every sum has a fixed order and every CTA forms bit-identical totals.
//
// Measured, us per iteration (50-iteration solves, launch included), streaming kernel -> this one:
//   Tet4 8 nodes 4.2 -> 0.85, 81 6.9 -> 1.2, 425 8.4 -> 2.4, 1,000 11.4 -> 2.4, 4,913 10.3 -> 3.7, 15,625 10.5 -> 4.1,
//   50,653 11.2 -> 5.7, 117,649 13.5 -> 10.1, 151,686 19.8 -> 13.2; Hex8 27 nodes 9.4 -> 1.2, 1,000 14.5 -> 2.6, 5,184
//   13.4 -> 3.9, 24,389 13.2 -> 4.8, 35,937 13.2 -> 5.8, 51,578 14.0 -> 7.4, 68,921 14.4 -> 8.8, 117,649 25.5..27.5 -> 21.6.
// What remains is the meeting (2.4 us of a grid, 1.0 of a cluster): at 5,184 Hex8 nodes most warps wait at the CTA
// barrier that follows it, 11% of the issue slots and 10% of the shared-memory pipe are used.  From 30,000 nodes come
// the columns read from L2: 44 MB an iteration at 68,921 nodes, where the product's shared wavefronts take 2 us.
#include <algorithm>
#include <vector>

#include "fem_grid.cuh"

namespace fem {
namespace {

constexpr int kSmemLimit = 227 * 1024 - 1024;  // dynamic: the kernel's static variables take a part of the first 1 KB
constexpr int kBlockBytes = 16 + 16 + 4 + 2;      // one resident block: values and local column
constexpr int kColumnBytes = kBlockBytes * kSlice;  // one resident block column of a slice
constexpr float kPredictFloor = 0.01f;
// A predicted rr1 carries the sums' rounding times at most (2 / sqrt(rr1 / rr) + 1)^2 = 441 at that floor: within this
// factor of the threshold it does not decide the stop, the sum itself does.
constexpr float kStopMargin = 1.01f;

// Scalars of the solve, formed by one thread from float totals (float32, like the reference's dot
// products; FP64 is far slower here and sits on every iteration's critical path: a quotient of two
// floats rounds to the same float either way, and the predictions are summed with their rounding
// errors).  floor_rr is the largest float that is at most tol^2 ||b||^2, so rr > floor_rr decides
// as the exact comparison does.
struct OcState {
    float rz, rr, bb, floor_rr;
    float scale, alpha, beta;
    int active, iters, again;
};

// c + b x + a x^2 for floats, with the rounding errors of every step carried along.
__device__ __forceinline__ float quadratic(float a, float b, float c, float x) {
    const float p = a * x, ep = fmaf(a, x, -p);  // a x = p + ep
    const float s = p + b, v = s - p, es = (p - (s - v)) + (b - v);  // p + b = s + es
    const float lo = ep + es;
    const float t = s * x, et = fmaf(s, x, -t);
    const float u = c + t, w = u - c, eu = (c - (u - w)) + (t - w);
    return u + (eu + fmaf(lo, x, et));
}

// Byte offsets of a CTA's dynamic shared memory; one definition for the kernel and the host.
// `own` is set in the variant that keeps matrix blocks in registers: its rows' x and inverse diagonal
// blocks are in shared memory instead.
struct OcLayout {
    int box, pb, part, own, halo, red, mat;  // mat: resident blocks (four planes)
};
constexpr int kOwnFloats = 12;
constexpr int kMaxCluster = 16;
__host__ __device__ __forceinline__ OcLayout oc_layout(int ns, int parts, int nhalo, bool own) {
    OcLayout l;
    const int rows = ns * kSlice;
    l.box = 0;  // first: a CTA writes its peers' boxes at the offset of its own, and the rest varies by CTA
    l.pb = l.box + 2 * kMaxCluster * 8 * 4;
    l.part = l.pb + (rows + nhalo) * 12;  // x, y and z planes
    l.own = l.part + (parts - 1) * rows * 12;
    l.halo = l.own + (own ? rows * kOwnFloats * 4 : 0);
    l.red = (l.halo + nhalo * 4 + 15) & ~15;
    l.mat = l.red + 32 * 8 * 4;
    return l;
}
__host__ __device__ __forceinline__ int oc_parts(int warps, int ns) { return ns > 0 ? max(1, warps / ns) : 1; }

constexpr int kTeamWords = 64, kTeamTicket = 32;  // counter and ticket on lines of their own
static_assert(kTeamWords * sizeof(unsigned) == kTeamBarrierBytes, "the host's allocation");

struct OcArgs {
    const float4* __restrict__ valA;
    const float4* __restrict__ valB;
    const float* __restrict__ valC;
    const unsigned short* __restrict__ lcol;  // [nsell] local column of each stored block
    const int* __restrict__ slice_ptr;
    const int2* __restrict__ slice_meta;
    const unsigned* __restrict__ row_info;
    const float* __restrict__ minv;
    const int* __restrict__ slice0;    // [grid+1] first slice of each CTA
    const int4* __restrict__ team;     // [grid] (first CTA, CTAs, scene, -) of the CTA's team
    const int2* __restrict__ kres;     // [nslices] (block columns in shared memory, the first one's place there)
    const int* __restrict__ halo_ptr;  // [grid+1]
    const int* __restrict__ halo;      // halo columns (node ids), per CTA ascending
    const float4* __restrict__ v4;
    const float4* __restrict__ q4;
    const float4* __restrict__ x4;  // packed warm start
    const float* __restrict__ rest;
    const int* __restrict__ spring_ptr;
    const int* __restrict__ spring_ent;
    const int* __restrict__ spring_idx;
    const float* __restrict__ spring_kd;
    float* f_ws;
    float* dv;
    float* q_out;
    float* v_out;
    float4* rec0;  // [3P] records (z, p, t), two alternating buffers
    float4* rec1;
    float* part;  // [2][grid][8]
    unsigned* barrier;  // [scenes][kTeamWords] a team's barrier counter and exit ticket
    int* status;
    SceneStats* scene_stats;
    long long* cum_iters;
    float* resid_max;
    int maxiter;
    float tol;
    float dt;
    long long limit_ns;
    int write_state;
    const float* solve_rhs;
    int solve_warm;
};

// The owner's and every reader's next search direction.
__device__ __forceinline__ float3 next_direction(float3 z, float3 t, float3 p, float alpha, float beta) {
    return f3(fmaf(beta, p.x, fmaf(-alpha, t.x, z.x)), fmaf(beta, p.y, fmaf(-alpha, t.y, z.y)),
              fmaf(beta, p.z, fmaf(-alpha, t.z, z.z)));
}

__device__ __forceinline__ float3 mul9(const float (&m)[9], float3 r) {
    return f3(m[0] * r.x + m[1] * r.y + m[2] * r.z, m[3] * r.x + m[4] * r.y + m[5] * r.z,
              m[6] * r.x + m[7] * r.y + m[8] * r.z);
}

// Per-thread constants of the product: this warp's slice and its share of the slice's columns,
// q, q + step, q + 2 step, ... -- the first kRegs of them in registers, the next ones in shared memory,
// the rest (kHybrid) in L2.
template <int kRegs>
struct Share {
    float m[kRegs > 0 ? kRegs : 1][9];
    int col[kRegs > 0 ? kRegs : 1];  // local columns of the register blocks
    const float4* A;                 // shared planes, this lane's block of column 0
    const float4* B;
    const float* C;
    const unsigned short* L;
    int len, kshared;  // this row's columns; the slice's columns below kshared are on chip
    int q, step;
    size_t e0;  // SELL entry of the lane's column 0
};

// Three planes of vector entries in shared memory (a float3 gather of consecutive columns takes three
// conflict-free wavefronts, a float4 one four).
struct Planes {
    float *x, *y, *z;
    __device__ __forceinline__ float3 get(int i) const { return f3(x[i], y[i], z[i]); }
    __device__ __forceinline__ void set(int i, float3 v) const {
        x[i] = v.x;
        y[i] = v.y;
        z[i] = v.z;
    }
};

// This warp's part of sum_k A_k (pb[col_k] - origin).
template <int kRegs, bool kHybrid, bool kDiff>
__device__ __forceinline__ float3 product_part(const OcArgs& a, const Share<kRegs>& s, const Planes& pb, float3 origin) {
    float3 acc = f3(0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < kRegs; ++i) {  // blocks past the row's end are zero
        float3 p = pb.get(s.col[i]);
        if (kDiff) p = p - origin;
        const float* m = s.m[i];
        acc = acc + f3(m[0] * p.x + m[1] * p.y + m[2] * p.z, m[3] * p.x + m[4] * p.y + m[5] * p.z,
                       m[6] * p.x + m[7] * p.y + m[8] * p.z);
    }
    int k = s.q + kRegs * s.step;
    const int ks = kHybrid ? min(s.len, s.kshared) : s.len;
#pragma unroll 2
    for (; k < ks; k += s.step) {
        const int i = k * kSlice;
        float3 p = pb.get(s.L[i]);
        if (kDiff) p = p - origin;
        acc = acc + bmul(s.A[i], s.B[i], s.C[i], p);
    }
    if (kHybrid) {
#pragma unroll 2
        for (; k < s.len; k += s.step) {
            const size_t e = s.e0 + (size_t)k * kSlice;
            const float4 A = __ldg(a.valA + e), B = __ldg(a.valB + e);
            const float C = __ldg(a.valC + e);
            float3 p = pb.get(__ldg(a.lcol + e));
            if (kDiff) p = p - origin;
            acc = acc + bmul(A, B, C, p);
        }
    }
    return acc;
}

// How the CTAs of a launch meet: alone, as one thread-block cluster (totals exchanged through
// distributed shared memory, one hardware cluster barrier per reduction: 1.0 us with 16 CTAs, the
// exchange of records through L2 included, against 1.7 us for a counter barrier of as many CTAs), or
// as a cooperative grid around a counter in global memory (2.4 us with 152).
enum Meet { kAlone, kCluster, kGrid, kTeams };  // kTeams: several such grids in one launch, one per scene

__device__ __forceinline__ void store_remote(const float* p, unsigned rank, float v) {
    const unsigned local = static_cast<unsigned>(__cvta_generic_to_shared(p));
    asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %0, %1;\n\t"
                 "st.shared::cluster.f32 [r], %2;\n\t}" ::"r"(local), "r"(rank), "f"(v) : "memory");
}
// The aligned forms are executed by whole warps together, and callers come from loops whose trip counts differ
// between lanes (a cluster's size and a halo's length are any number): the warp meets first.
__device__ __forceinline__ void cluster_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The eight values of `acc` over lanes with equal lane & 7 (component 7: maximum when kMax).
template <bool kMax>
__device__ __forceinline__ float fold_groups(float acc, int c) {
#pragma unroll
    for (int off = 8; off < 32; off <<= 1) {
        const float o = __shfl_xor_sync(0xffffffffu, acc, off);
        acc = (kMax && c == 7) ? fmaxf(acc, o) : acc + o;
    }
    return acc;
}

// Sums of v[0..6] and (kMax) the maximum of v[7] over all rows.  Each owner warp folds its eight
// values over its lanes (one exchange halves the values a lane carries), warp 0 adds the warps and
// then the CTAs' totals; lane 0 runs upd(totals).  Entered by the whole CTA; false after a wait that
// ran out (kGrid only).
template <Meet kMeet, bool kMax, class Update>
__device__ __forceinline__ bool reduce8(const OcArgs& a, int4 team, float (&v)[8], int ns, float* red, float* box,
                                        unsigned& epoch, int* s_ok, Update upd) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = lane & 7;
    if (warp < ns) {
        const float m = kMax ? warp_max(v[7]) : 0.0f;
        float w4[4], w2[2], w;
        const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            w4[i] = (b4 ? v[i + 4] : v[i]) + __shfl_xor_sync(0xffffffffu, b4 ? v[i] : v[i + 4], 16);
#pragma unroll
        for (int i = 0; i < 2; ++i)
            w2[i] = (b3 ? w4[i + 2] : w4[i]) + __shfl_xor_sync(0xffffffffu, b3 ? w4[i] : w4[i + 2], 8);
        w = (b2 ? w2[1] : w2[0]) + __shfl_xor_sync(0xffffffffu, b2 ? w2[0] : w2[1], 4);
        w += __shfl_xor_sync(0xffffffffu, w, 2);
        w += __shfl_xor_sync(0xffffffffu, w, 1);
        const int cv = lane >> 2;  // the value this lane's group of four holds
        if ((lane & 3) == 0) red[warp * 8 + cv] = (kMax && cv == 7) ? m : w;
    }
    __syncthreads();
    float acc = 0.0f;
    if (warp == 0) {
        for (int w = lane >> 3; w < ns; w += 4) acc = (kMax && c == 7) ? fmaxf(acc, red[w * 8 + c]) : acc + red[w * 8 + c];
        acc = fold_groups<kMax>(acc, c);
    }
    int ok = 1;
    if (kMeet == kCluster) {
        // two sets of boxes: a CTA writes a set again only after the barrier that follows its readers
        float* mine = box + (epoch & 1u) * kMaxCluster * 8;
        epoch += 1;
        if (warp == 0)
            for (unsigned r = lane >> 3; r < gridDim.x; r += 4) store_remote(mine + blockIdx.x * 8 + c, r, acc);
        cluster_barrier();
        if (warp == 0) {
            acc = 0.0f;
            for (unsigned r = lane >> 3; r < gridDim.x; r += 4)
                acc = (kMax && c == 7) ? fmaxf(acc, mine[r * 8 + c]) : acc + mine[r * 8 + c];
            acc = fold_groups<kMax>(acc, c);
        }
    }
    if (warp == 0) {
        if (kMeet == kGrid || (kMeet == kTeams && team.y > 1)) {
            const int G = team.y;
            float* buf = a.part + ((size_t)(epoch & 1u) * gridDim.x + team.x) * 8;
            if (lane < 8) buf[(blockIdx.x - team.x) * 8 + lane] = acc;
            __syncwarp();
            if (lane == 0) ok = arrive_and_wait(a.barrier + team.z * kTeamWords, G, epoch, a.status, a.limit_ns);
            ok = __shfl_sync(0xffffffffu, ok, 0);
            epoch = __shfl_sync(0xffffffffu, epoch, 0);
            __syncwarp();  // orders what lane 0 has acquired before the other lanes' loads (a shuffle does not)
            if (ok) {  // lane: half (lane & 1) of the records of CTAs (lane >> 1), (lane >> 1) + 16, ...
                const float4* b4 = reinterpret_cast<const float4*>(buf);
                float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
                constexpr int kBatch = 10;
                for (int g0 = lane >> 1; g0 < G; g0 += 16 * kBatch) {
                    float4 t[kBatch];
#pragma unroll
                    for (int u = 0; u < kBatch; ++u) {
                        const int g = g0 + 16 * u;
                        t[u] = g < G ? __ldcg(b4 + 2 * g + (lane & 1)) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                    for (int u = 0; u < kBatch; ++u) {
                        s.x += t[u].x;
                        s.y += t[u].y;
                        s.z += t[u].z;
                        s.w = (kMax && (lane & 1)) ? fmaxf(s.w, t[u].w) : s.w + t[u].w;
                    }
                }
#pragma unroll
                for (int off = 2; off < 32; off <<= 1) {
                    s.x += __shfl_xor_sync(0xffffffffu, s.x, off);
                    s.y += __shfl_xor_sync(0xffffffffu, s.y, off);
                    s.z += __shfl_xor_sync(0xffffffffu, s.z, off);
                    const float o = __shfl_xor_sync(0xffffffffu, s.w, off);
                    s.w = (kMax && (lane & 1)) ? fmaxf(s.w, o) : s.w + o;
                }
                // lanes 0..7 take components 0..7
                const int src = c >> 2;
                const float e0 = __shfl_sync(0xffffffffu, s.x, src), e1 = __shfl_sync(0xffffffffu, s.y, src);
                const float e2 = __shfl_sync(0xffffffffu, s.z, src), e3 = __shfl_sync(0xffffffffu, s.w, src);
                acc = (c & 3) == 0 ? e0 : ((c & 3) == 1 ? e1 : ((c & 3) == 2 ? e2 : e3));
            }
        }
        float T[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) T[k] = __shfl_sync(0xffffffffu, acc, k);
        if (lane == 0) {
            if (ok) upd(T);
            *s_ok = ok;
        }
    }
    __syncthreads();
    return *s_ok != 0;
}

// Sums of v[i] over the rows of a CTA that is alone, formed by every warp from the owner warps' sums: one CTA
// barrier.  `slots` holds 32 N floats; a caller alternates them, as a warp may still be reading the last call's.
template <int N>
__device__ __forceinline__ void cta_sums(float (&v)[N], int ns, float* slots) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < ns) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const float w = warp_sum(v[i]);
            if (lane == 0) slots[32 * i + warp] = w;
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = warp_sum(lane < ns ? slots[32 * i + lane] : 0.0f);
}

template <int kRegs, int kThreads, bool kHybrid, Meet kMeet>
__global__ void __launch_bounds__(kThreads, 1) onchip_pcg_kernel(OcArgs a) {
    chained_start();
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ OcState st;
    __shared__ int s_ok;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
    // a constant of the launch where there is one team (its registers cost the 64-register variant 9%)
    const int4 team = kMeet == kTeams ? a.team[blockIdx.x] : make_int4(0, (int)gridDim.x, 0, 0);
    const int first = a.slice0[blockIdx.x], ns = a.slice0[blockIdx.x + 1] - first;
    const int h0 = a.halo_ptr[blockIdx.x], nhalo = a.halo_ptr[blockIdx.x + 1] - h0;
    const int Q = oc_parts(W, ns), rows = ns * kSlice;
    const OcLayout lay = oc_layout(ns, Q, nhalo, kRegs > 0);
    Planes pb;
    pb.x = reinterpret_cast<float*>(smem + lay.pb);
    pb.y = pb.x + rows + nhalo;
    pb.z = pb.y + rows + nhalo;
    float* part = reinterpret_cast<float*>(smem + lay.part);
    int* hid = reinterpret_cast<int*>(smem + lay.halo);
    float* red = reinterpret_cast<float*>(smem + lay.red);
    float* box = reinterpret_cast<float*>(smem + lay.box);
    float* own = reinterpret_cast<float*>(smem + lay.own) + (threadIdx.x < (unsigned)rows ? threadIdx.x : 0);
    unsigned epoch = 0;

    // This warp's slice and its share of the columns; copy the resident ones (only this thread reads
    // back what it copies, so no barrier is needed for them).
    const int t = ns > 0 ? warp % ns : 0, q = ns > 0 ? warp / ns : Q;
    const bool works = q < Q;
    const bool owner = warp < ns;
    Share<kRegs> sh;
    int row = 0, lr = t * kSlice + lane;
    bool live = false, fixed = false;
    {
        int cols = 0;  // shared columns of the CTA (plane sizes)
        if (ns > 0) {
            const int2 kl = a.kres[first + ns - 1];
            cols = kl.x + kl.y;
        }
        float4* sA = reinterpret_cast<float4*>(smem + lay.mat);
        float4* sB = sA + (size_t)cols * kSlice;
        float* sC = reinterpret_cast<float*>(sB + (size_t)cols * kSlice);
        unsigned short* sL = reinterpret_cast<unsigned short*>(sC + (size_t)cols * kSlice);
        sh.len = 0;
        sh.kshared = 0;
        sh.q = q;
        sh.step = Q;
        sh.e0 = 0;
        sh.A = sA;
        sh.B = sB;
        sh.C = sC;
        sh.L = sL;
#pragma unroll
        for (int i = 0; i < (kRegs > 0 ? kRegs : 1); ++i) {
            sh.col[i] = lr;
#pragma unroll
            for (int k = 0; k < 9; ++k) sh.m[i][k] = 0.0f;
        }
        if (works && ns > 0) {
            const int sl = first + t;
            const int2 m = a.slice_meta[sl], kr = a.kres[sl];
            live = lane < m.y;
            row = m.x + lane;
            const unsigned info = live ? a.row_info[row] : 0u;
            fixed = (info & kFixedBit) != 0;
            sh.len = fixed ? 0 : (int)(info & ~kFixedBit);
            sh.e0 = (size_t)a.slice_ptr[sl] * kSlice + lane;
#pragma unroll
            for (int i = 0; i < kRegs; ++i) {
                const int k = q + i * Q;
                if (k < sh.len) {
                    const size_t e = sh.e0 + (size_t)k * kSlice;
                    const float4 A = __ldg(a.valA + e), B = __ldg(a.valB + e);
                    sh.m[i][0] = A.x; sh.m[i][1] = A.y; sh.m[i][2] = A.z; sh.m[i][3] = A.w;
                    sh.m[i][4] = B.x; sh.m[i][5] = B.y; sh.m[i][6] = B.z; sh.m[i][7] = B.w;
                    sh.m[i][8] = __ldg(a.valC + e);
                    sh.col[i] = __ldg(a.lcol + e);
                }
            }
            const int k0 = kRegs * Q;  // first column in shared memory
            sh.kshared = k0 + kr.x;
            const int at = (kr.y - k0) * kSlice + lane;
            sh.A = sA + at;
            sh.B = sB + at;
            sh.C = sC + at;
            sh.L = sL + at;
            const int kn = min(sh.len, sh.kshared);
#pragma unroll 4
            for (int k = q + k0; k < kn; k += Q) {
                const size_t e = sh.e0 + (size_t)k * kSlice;
                sA[at + k * kSlice] = __ldg(a.valA + e);
                sB[at + k * kSlice] = __ldg(a.valB + e);
                sC[at + k * kSlice] = __ldg(a.valC + e);
                sL[at + k * kSlice] = __ldg(a.lcol + e);
            }
        }
        for (int c = threadIdx.x; c < nhalo; c += blockDim.x) hid[c] = a.halo[h0 + c];
    }
    live = live && owner;

    // One product into the owner's registers: the caller has filled pb.
    auto finish = [&](float3 acc) {  // add the other warps' parts of the owner's row, in order
        if (works && q > 0) {
            float* o = part + (size_t)(q - 1) * 3 * rows + lr;
            o[0] = acc.x;
            o[rows] = acc.y;
            o[2 * rows] = acc.z;
        }
        __syncthreads();
        if (owner)
            for (int u = 0; u + 1 < Q; ++u) {
                const float* o = part + (size_t)u * 3 * rows + lr;
                acc = acc + f3(o[0], o[rows], o[2 * rows]);
            }
        return acc;
    };
    auto fill = [&](const float4* src) {
        if (owner) pb.set(lr, live ? xyz(src[row]) : f3(0.f, 0.f, 0.f));
        for (int c = threadIdx.x; c < nhalo; c += blockDim.x) pb.set(rows + c, xyz(src[hid[c]]));
        __syncthreads();
    };
    const float3 zero = f3(0.f, 0.f, 0.f);
    if (kMeet == kCluster) cluster_barrier();  // halo ids, and every CTA has started
    else __syncthreads();                      // halo ids

    // ---- right-hand side (predictor, spring damping, projection) and initial residual
    float3 rhs = zero, x = zero, r = zero;
    const bool step_mode = a.solve_rhs == nullptr;
    if (step_mode) {
        fill(a.v4);
        const float3 cv = finish(works ? product_part<kRegs, kHybrid, true>(a, sh, pb, pb.get(lr)) : zero);
        if (live && !fixed) {
            rhs = load3(a.f_ws, row) - cv;
            for (int e = a.spring_ptr[row]; e < a.spring_ptr[row + 1]; ++e) {
                const int ent = a.spring_ent[e], s = ent >> 1;
                const int ia = a.spring_idx[2 * s], ib = a.spring_idx[2 * s + 1];
                if (ia < 0 || ib < 0) continue;
                const float3 corr = (xyz(a.v4[ia]) - xyz(a.v4[ib])) * (a.dt * a.spring_kd[s]);
                rhs = (ent & 1) ? rhs - corr : rhs + corr;
            }
        }
        if (live) store3(a.f_ws, row, rhs);
    } else if (live && !fixed) {
        rhs = load3(a.solve_rhs, row);
    }
    r = rhs;
    if (step_mode || a.solve_warm) {
        fill(a.x4);
        const float3 ax = finish(works ? product_part<kRegs, kHybrid, false>(a, sh, pb, zero) : zero);
        if (live) {
            x = pb.get(lr);
            r = rhs - ax;
            if (fixed) r = zero;
        }
    }
    // the row's inverse diagonal block and x: registers, or (when the matrix has those) shared memory
    float mi[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) mi[k] = live ? a.minv[9 * (size_t)row + k] : 0.0f;
    if (kRegs > 0 && owner) {
#pragma unroll
        for (int k = 0; k < 9; ++k) own[(3 + k) * rows] = mi[k];
    }
    auto precondition = [&](float3 u) {
        if (kRegs > 0) {
            if (!owner) return zero;
            const float* m = own + 3 * rows;
            return f3(m[0] * u.x + m[rows] * u.y + m[2 * rows] * u.z,
                      m[3 * rows] * u.x + m[4 * rows] * u.y + m[5 * rows] * u.z,
                      m[6 * rows] * u.x + m[7 * rows] * u.y + m[8 * rows] * u.z);
        }
        return mul9(mi, u);
    };
    auto set_x = [&](float3 u) {
        if (kRegs > 0) {
            if (owner) {
                own[0] = u.x;
                own[rows] = u.y;
                own[2 * rows] = u.z;
            }
        } else {
            x = u;
        }
    };
    auto get_x = [&]() { return kRegs > 0 ? (owner ? f3(own[0], own[rows], own[2 * rows]) : zero) : x; };
    set_x(x);
    float3 z = precondition(r), p = zero, s = zero, tt = zero;
    auto publish = [&](float4* rec) {
        if (kMeet != kAlone && live) {
            rec[3 * (size_t)row] = make_float4(z.x, z.y, z.z, p.x);
            rec[3 * (size_t)row + 1] = make_float4(p.y, p.z, tt.x, tt.y);
            rec[3 * (size_t)row + 2] = make_float4(tt.z, 0.f, 0.f, 0.f);
        }
    };
    auto start = [&](const float* T) {
        st.rr = T[0];
        st.rz = T[1];
        st.bb = T[2];
        st.floor_rr = __double2float_rd((double)a.tol * (double)a.tol * (double)T[2]);
        st.iters = 0;
        st.alpha = 0.0f;
        st.beta = 0.0f;
        st.again = 0;
        st.active = (st.rr > st.floor_rr) && (a.maxiter > 0);
        if (!isfinite(st.rr)) {
            st.active = 0;
            atomicOr(a.status, kStatusNonFinite);
        }
    };
    bool ok;
    {
        publish(a.rec0);
        float v[8] = {dot3(r, r), dot3(r, z), dot3(rhs, rhs), 0.f, 0.f, 0.f, 0.f,
                      fmaxf(fabsf(rhs.x), fmaxf(fabsf(rhs.y), fabsf(rhs.z)))};
        ok = reduce8<kMeet, true>(a, team, v, ns, red, box, epoch, &s_ok, [&](const float* T) {
            if (T[7] == 0.0f) {  // b = 0: the warm start is cleared (x = 0 solves it)
                const float none[8] = {0.f, 0.f, T[2], 0.f, 0.f, 0.f, 0.f, 0.f};
                start(none);
                st.scale = 0.0f;
            } else {
                start(T);
                st.scale = rhs_scale(T[7]);
            }
        });
    }
    if (ok) {
        const float scale = st.scale;
        if (scale == 0.0f) {
            set_x(zero);
            r = zero;
        } else if (scale != 1.0f) {  // a tiny right-hand side: the sums again on the normalised system
            set_x(get_x() * scale);
            r = r * scale;
            z = precondition(r);
            const float3 b = rhs * scale;
            publish(a.rec0);
            float v[8] = {dot3(r, r), dot3(r, z), dot3(b, b), 0.f, 0.f, 0.f, 0.f, 0.f};
            ok = reduce8<kMeet, false>(a, team, v, ns, red, box, epoch, &s_ok, start);
        }
    }

    // ---- CG iterations
    const bool alone = kMeet == kAlone || (kMeet == kTeams && team.y == 1);
    if (alone) {
        // One CTA, no halo: the two reductions of standard CG are CTA barriers, so every scalar is the sum itself.
        // (With predicted ones, bodies of 8 to 164 nodes, which converge in steep last steps, ended 1.5 to 3 times as
        // far from the 64-bit iterates as the streaming kernel's, and took up to 0.7 iterations more.)
        float rz = st.rz, rr = st.rr;
        int n = 0;
        p = z;
        for (bool go = st.active; go;) {
            if (owner) pb.set(lr, p);
            __syncthreads();
            s = finish(works ? product_part<kRegs, kHybrid, false>(a, sh, pb, zero) : zero);
            float ps[1] = {dot3(p, s)};
            cta_sums(ps, ns, red);
            if (owner) {
                const float al = rz / ps[0];
                const float3 xo = get_x();
                set_x(f3(fmaf(al, p.x, xo.x), fmaf(al, p.y, xo.y), fmaf(al, p.z, xo.z)));
                r = f3(fmaf(-al, s.x, r.x), fmaf(-al, s.y, r.y), fmaf(-al, s.z, r.z));
                z = precondition(r);
            }
            float v[2] = {dot3(r, r), dot3(r, z)};
            cta_sums(v, ns, red + 32);
            const float be = v[1] / rz;
            rr = v[0];
            rz = v[1];
            p = f3(fmaf(be, p.x, z.x), fmaf(be, p.y, z.y), fmaf(be, p.z, z.z));
            ++n;
            go = isfinite(rr) && rr > st.floor_rr && n < a.maxiter;
        }
        p = zero;  // x is complete: nothing is left for the epilogue to add
        if (threadIdx.x == 0) {
            st.iters = n;
            st.rr = rr;
            if (!isfinite(rr)) atomicOr(a.status, kStatusNonFinite);
        }
    }
    for (int it = 0; !alone && ok && st.active; ++it) {
        const float4* rec = (it & 1) ? a.rec1 : a.rec0;
        const float al = st.alpha, be = st.beta;
        for (int c = threadIdx.x; c < nhalo; c += blockDim.x) {
            const float4* o = rec + 3 * (size_t)hid[c];
            const float4 o0 = o[0], o1 = o[1];
            const float o2 = reinterpret_cast<const float*>(o + 2)[0];
            pb.set(rows + c, next_direction(xyz(o0), f3(o1.z, o1.w, o2), f3(o0.w, o1.x, o1.y), al, be));
        }
        if (owner) {
            const float3 pn = next_direction(z, tt, p, al, be);
            pb.set(lr, pn);
            const float3 xo = get_x();
            set_x(f3(fmaf(al, p.x, xo.x), fmaf(al, p.y, xo.y), fmaf(al, p.z, xo.z)));
            r = f3(fmaf(-al, s.x, r.x), fmaf(-al, s.y, r.y), fmaf(-al, s.z, r.z));
            z = precondition(r);
            p = pn;
        }
        __syncthreads();
        s = finish(works ? product_part<kRegs, kHybrid, false>(a, sh, pb, zero) : zero);  // zero at fixed rows, as p is
        tt = precondition(s);
        publish((it & 1) ? a.rec0 : a.rec1);
        {
            float v[8] = {dot3(p, s), dot3(z, s), dot3(tt, s), dot3(r, z), dot3(r, r), dot3(r, s), dot3(s, s), 0.f};
            ok = reduce8<kMeet, false>(a, team, v, ns, red, box, epoch, &s_ok, [&](const float* T) {
                const float rz = T[3], rr = T[4], alpha = rz / T[0];
                const float rz1 = quadratic(T[2], -2.0f * T[1], rz, alpha);
                const float rr1 = quadratic(T[6], -2.0f * T[5], rr, alpha);
                st.alpha = alpha;
                st.beta = rz1 / rz;
                st.rr = rr1;
                st.rz = rz;
                st.iters += 1;
                st.again = rz1 < kPredictFloor * rz || rr1 < kPredictFloor * rr ||
                           (rr1 <= kStopMargin * st.floor_rr && kStopMargin * rr1 > st.floor_rr);
                st.active = (rr1 > st.floor_rr) && (st.iters < a.maxiter);
                if (!isfinite(rr1)) {
                    st.active = 0;
                    st.again = 0;
                    atomicOr(a.status, kStatusNonFinite);
                }
            });
        }
        if (ok && st.again) {  // the predictions cancelled, or are too close to the threshold: the sums themselves
            const float a1 = st.alpha;
            const float3 r1 = f3(fmaf(-a1, s.x, r.x), fmaf(-a1, s.y, r.y), fmaf(-a1, s.z, r.z));
            float v[8] = {dot3(r1, precondition(r1)), dot3(r1, r1), 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            ok = reduce8<kMeet, false>(a, team, v, ns, red, box, epoch, &s_ok, [&](const float* T) {
                st.beta = T[0] / st.rz;
                st.rr = T[1];
                st.active = (st.rr > st.floor_rr) && (st.iters < a.maxiter);
                if (!isfinite(st.rr)) {
                    st.active = 0;
                    atomicOr(a.status, kStatusNonFinite);
                }
            });
        }
    }

    // ---- the residual that is reported: the sum over the final r, not its prediction.  Nobody waits for it: a CTA
    // leaves its part with its exit ticket, and the last one to take a ticket adds them, in a fixed order.  Both are
    // under way while the epilogue stores (after it, behind a fence for its stores, they took 3.5 us; as one more
    // reduction 1.7 in a cluster and 3.6 in a grid).
    const bool several = kMeet != kAlone && team.y > 1;
    float* const parts = a.part + ((size_t)(epoch & 1u) * gridDim.x + team.x) * 8;  // as a next reduction's
    unsigned* const words = a.barrier + team.z * kTeamWords;
    float rr_end = st.rr;
    unsigned left = 0;  // the CTAs that left before this one
    if (several) {
        if (warp < ns) {
            const float al = st.alpha;
            const float3 r1 = f3(fmaf(-al, s.x, r.x), fmaf(-al, s.y, r.y), fmaf(-al, s.z, r.z));
            const float rr = warp_sum(dot3(r1, r1));
            if (lane == 0) red[warp] = rr;
        }
        __syncthreads();
        if (warp == 0) {
            const float rr = warp_sum(lane < ns ? red[lane] : 0.0f);
            if (lane == 0) {
                parts[(blockIdx.x - team.x) * 8] = rr;
                asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;"
                             : "=r"(left)
                             : "l"(words + kTeamTicket)
                             : "memory");
            }
        }
    }

    // ---- epilogue: the last update of x, restore the scale, integrate, fixed restore
    if (ok && live) {
        const float al = st.alpha, sc = st.scale == 0.0f ? 1.0f : st.scale;
        const float3 xo = get_x();
        float3 dv = f3(fmaf(al, p.x, xo.x), fmaf(al, p.y, xo.y), fmaf(al, p.z, xo.z));
        dv = f3(dv.x / sc, dv.y / sc, dv.z / sc);
        store3(a.dv, row, dv);
        if (a.write_state) {
            float3 v = xyz(a.v4[row]) + dv;
            float3 qn = xyz(a.q4[row]) + v * a.dt;
            if (fixed) {
                qn = load3(a.rest, row);
                v = zero;
            }
            store3(a.q_out, row, qn);
            store3(a.v_out, row, v);
        }
    }
    if (warp == 0) {
        const bool last = !several || __shfl_sync(0xffffffffu, left, 0) == (unsigned)team.y - 1;
        if (several && last) {
            __syncwarp();  // the parts that lane 0 has acquired, for every lane
            rr_end = 0.0f;
            for (int g = lane; g < team.y; g += 32) rr_end += __ldcg(parts + 8 * g);
            rr_end = warp_sum(rr_end);
            if (lane == 0) {  // and clears the team's barrier for the next launch: no memset per solve
                words[0] = 0u;
                words[kTeamTicket] = 0u;
            }
        }
        if (ok && last && lane == 0) {
            SceneStats o;
            o.iterations = st.iters;
            o.rr = rr_end;
            o.bb = st.bb;
            o.converged = rr_end <= st.floor_rr;
            a.scene_stats[team.z] = o;
            // an atomic has no load to wait for at the kernel's end (0.3 us)
            atomicAdd(reinterpret_cast<unsigned long long*>(a.cum_iters + team.z), (unsigned long long)st.iters);
            // running max of the relative residual (non-negative floats order like their bit patterns)
            float rel = st.bb > 0.0f ? (float)sqrt((double)rr_end / (double)st.bb) : 0.0f;
            if (!isfinite(rel)) rel = 1.0e30f;
            atomicMax(reinterpret_cast<int*>(a.resid_max + (step_mode ? 0 : 1)), __float_as_int(rel));
        }
    }
}

using OcKernel = void (*)(OcArgs);
// Up to 16 slices per CTA run in 512 threads of 128 registers, kOcRegs blocks per thread of which are
// matrix (the product is bound by shared-memory wavefronts: a register block costs the three of its
// gather, a shared one fourteen; 5, 6 and 7 blocks spill: 3.9, 4.3 and 4.7 us per iteration against 3.8
// on 5,184 nodes); more slices (one owner thread per row) in 1024 threads of 64.
constexpr int kOcRegs = 4, kOcWideWarps = 16;
// Where the launches cross, in stored block columns of all slices (us per iteration on GB300, one CTA and a cluster):
//   Hex8 27 nodes (27 columns) 1.2 and 1.9, Tet4 180 (90) 1.7 and 2.1, Hex8 125 (108) 1.7 and 2.3, Tet4 252 (120) 1.8
//   and 2.1, Hex8 150 (135) 1.8 and 2.3, Hex8 180 (162) 2.1 and 2.2, Tet4 448 (210) 2.3 and 2.4, Hex8 245 (216) 2.45
//   and 2.3: the crossing is near 200, and the line, at 128, is where every body measured is faster alone;
//   a cluster of 16 reaches a grid's 3.4 near 2,000 columns (Hex8 74 slices, 1,998 columns: 3.22 and
//   3.39; Tet4 106 slices, 1,590: 3.16 and 3.34; Hex8 106 slices, 2,862: 3.85 and 3.47).
constexpr int64_t kAloneColumns = 128, kClusterColumns = 2000;
// Where the streaming kernel is the faster one although the rows fit (us per iteration, streaming and on chip):
//   a CTA reads a 48-byte record for every halo column, so a numbering without locality costs it more than the
//   streaming kernel, whose gathers are as many blocks as before.  Tet4 with nodes numbered at random: 42,875 nodes
//   (3,746 halo and 132 block columns a CTA) 12.3 and 9.5, 50,653 (4,589, 156) 12.5 and 14.0, 68,921 (6,207, 213) 13.5
//   and 17.7; Hex8 32,768 (5,169, 182) 14.8 and 13.8, 68,921 (10,964, 383) 18.0 and 25.7; numbers off by about 3,000
//   places: Tet4 68,921 (4,915, 213) 14.0 and 14.3, 148,877 (8,454, 459) 22.8 and 23.8, Hex8 68,921 (7,414, 383) 18.1
//   and 18.2.  The line through the crossings is kHaloBase + kHaloPerColumn x block columns;
//   the columns that are not on chip are read from L2 until they no longer stay there: Hex8 117,649 nodes (89 MB)
//   27.4 and 21.5, 125,000 (97 MB) 27.7 and 27.5, 132,651 (105 MB) 29.3 and 29.6, 140,608 (113 MB) 30.3 and 32.8.
constexpr int kHaloBase = 3000, kHaloPerColumn = 10;
constexpr double kL2Share = 0.7;
template <Meet kMeet>
OcKernel oc_kernel_for(int threads, bool hybrid) {
    if (threads <= 32 * kOcWideWarps)
        return hybrid ? onchip_pcg_kernel<kOcRegs, 512, true, kMeet> : onchip_pcg_kernel<kOcRegs, 512, false, kMeet>;
    constexpr Meet kWide = kMeet == kTeams ? kTeams : kGrid;
    return hybrid ? onchip_pcg_kernel<0, 1024, true, kWide> : onchip_pcg_kernel<0, 1024, false, kWide>;
}
OcKernel oc_kernel(int meet, int threads, bool hybrid) {
    switch (meet) {
        case kAlone: return oc_kernel_for<kAlone>(threads, hybrid);
        case kCluster: return oc_kernel_for<kCluster>(threads, hybrid);
        case kGrid: return oc_kernel_for<kGrid>(threads, hybrid);
        default: return oc_kernel_for<kTeams>(threads, hybrid);
    }
}

cudaLaunchAttribute cluster_attribute(int ctas) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = ctas;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    return attr;
}

}  // namespace

// Teams of CTAs for several scenes: the smallest number of slices per CTA that one wave holds, then the
// CTAs left over to the scenes with the most slices per CTA.  No teams when a CTA would need more than 32.
static void plan_teams(const Handle& h, int sms, OnchipPlan& plan) {
    std::vector<int> s0(h.nscenes + 1, 0);
    for (int sl = 0; sl < h.nslices; ++sl) s0[h.host_slice_scene[sl] + 1]++;
    for (int sc = 0; sc < h.nscenes; ++sc) s0[sc + 1] += s0[sc];
    auto slices = [&](int sc) { return s0[sc + 1] - s0[sc]; };
    int most = std::max(1, (h.nslices + sms - 1) / sms), used = 0;
    for (;; ++most) {
        if (most > 32) return;
        used = 0;
        for (int sc = 0; sc < h.nscenes; ++sc) used += (slices(sc) + most - 1) / most;
        if (used <= sms) break;
    }
    std::vector<int> ctas(h.nscenes);
    for (int sc = 0; sc < h.nscenes; ++sc) ctas[sc] = (slices(sc) + most - 1) / most;
    for (; used < sms; ++used) {
        int best = -1;
        for (int sc = 0; sc < h.nscenes; ++sc)
            if (ctas[sc] < slices(sc) &&
                (best < 0 || (int64_t)slices(sc) * ctas[best] > (int64_t)slices(best) * ctas[sc]))
                best = sc;
        if (best < 0) break;
        ++ctas[best];
    }
    for (int sc = 0; sc < h.nscenes; ++sc) {
        const int at = (int)plan.team.size();
        for (int c = 0; c < ctas[sc]; ++c) {
            plan.slice0.push_back(s0[sc] + (int)((int64_t)slices(sc) * c / ctas[sc]));
            plan.team.push_back(make_int4(at, ctas[sc], sc, 0));
        }
    }
    plan.slice0.push_back(h.nslices);
}

// Lays a handle out for the on-chip kernel: the CTAs' slices, their halo lists and local columns and
// the resident share of the columns.  Leaves plan.grid 0 when the rows do not fit.
void onchip_plan(const Handle& h, const OnchipInput& in, int sms, int64_t l2_bytes, OnchipPlan& plan) {
    plan = OnchipPlan{};
    if (h.nslices == 0 || h.nscenes > sms) return;
    int width = 0;
    int64_t columns = 0;
    for (int sl = 0; sl < h.nslices; ++sl) {
        const int w = h.host_slice_ptr[sl + 1] - h.host_slice_ptr[sl];
        width = std::max(width, w);
        columns += w;
    }
    const int wanted = std::max(1, (width + 3) / 4);  // warps per slice: about four columns each
    int grid = std::min(sms, h.nslices);
    plan.meet = kGrid;
    if (h.nscenes > 1) {
        plan.meet = kTeams;
        plan_teams(h, sms, plan);
        grid = (int)plan.team.size();
        if (grid == 0) return;
    } else {
        if (columns <= kAloneColumns && h.nslices <= kOcWideWarps) {
            grid = 1;
            plan.meet = kAlone;
        } else if (columns <= kClusterColumns && h.nslices <= kMaxCluster * kOcWideWarps) {
            grid = std::min(kMaxCluster, h.nslices);
            plan.meet = kCluster;
        }
        if ((h.nslices + grid - 1) / grid > (plan.meet == kGrid ? 32 : kOcWideWarps)) return;
        // contiguous runs balanced by stored blocks
        plan.slice0 = in.split(grid);
        plan.team.assign(grid, make_int4(0, grid, 0, 0));
    }
    int widest = 0;
    for (int c = 0; c < grid; ++c) widest = std::max(widest, plan.slice0[c + 1] - plan.slice0[c]);
    if (widest > 32) return;
    const int most = widest <= kOcWideWarps ? kOcWideWarps : 32, regs = widest <= kOcWideWarps ? kOcRegs : 0;
    const int warps = std::min(most, std::max(widest, std::max(4, widest * wanted)));
    plan.lcol.assign((size_t)h.nsell, 0);
    plan.kres.assign(h.nslices, make_int2(0, 0));
    plan.halo_ptr.assign(grid + 1, 0);
    std::vector<std::vector<int>> halos(grid);
    std::vector<char> fits(grid, 1);
    std::vector<int> bytes(grid, 0), partial(grid, 0), slow(grid, 0);
    std::vector<int64_t> streamed(grid, 0);  // block columns read from L2 in every iteration
    in.parallel(grid, [&](int64_t lo, int64_t hi) {
        std::vector<int> local(h.P, -1);
        for (int64_t c = lo; c < hi; ++c) {
            const int s0 = plan.slice0[c], s1 = plan.slice0[c + 1], ns = s1 - s0;
            std::vector<int>& halo = halos[c];
            if (ns == 0) continue;
            auto each = [&](auto&& fn) {
                for (int sl = s0; sl < s1; ++sl) {
                    const int base = h.host_slice_ptr[sl];
                    for (int l = 0; l < in.slice_meta[sl].y; ++l) {
                        const int r = in.slice_meta[sl].x + l;
                        for (int k = 0; k < (int)(in.row_info[r] & ~kFixedBit); ++k) fn((int64_t)(base + k) * kSlice + l);
                    }
                }
            };
            for (int sl = s0; sl < s1; ++sl)
                for (int l = 0; l < in.slice_meta[sl].y; ++l) local[in.slice_meta[sl].x + l] = (sl - s0) * kSlice + l;
            each([&](int64_t e) {
                const int j = in.scol[e];
                if (local[j] < 0) {
                    local[j] = 0;
                    halo.push_back(j);
                }
            });
            std::sort(halo.begin(), halo.end());
            for (size_t i = 0; i < halo.size(); ++i) local[halo[i]] = ns * kSlice + (int)i;
            const int ncols = ns * kSlice + (int)halo.size();
            if (ncols > 65535) fits[c] = 0;
            each([&](int64_t e) { plan.lcol[e] = (unsigned short)local[in.scol[e]]; });
            for (int sl = s0; sl < s1; ++sl)
                for (int l = 0; l < in.slice_meta[sl].y; ++l) local[in.slice_meta[sl].x + l] = -1;
            for (int j : halo) local[j] = -1;
            // resident columns: all of them, or a uniform share of every slice's
            const int fixed_bytes = oc_layout(ns, oc_parts(warps, ns), (int)halo.size(), regs > 0).mat;
            if (fixed_bytes > kSmemLimit) {
                fits[c] = 0;
                continue;
            }
            const int64_t room = (kSmemLimit - fixed_bytes) / kColumnBytes;
            const int in_regs = regs * oc_parts(warps, ns);  // columns of each slice kept in registers
            auto rest = [&](int sl) {
                return (int64_t)std::max(0, h.host_slice_ptr[sl + 1] - h.host_slice_ptr[sl] - in_regs);
            };
            int64_t total = 0, at = 0;
            for (int sl = s0; sl < s1; ++sl) total += rest(sl);
            for (int sl = s0; sl < s1; ++sl) {
                const int k = (int)(total > room ? rest(sl) * room / total : rest(sl));
                plan.kres[sl] = make_int2(k, (int)at);
                at += k;
            }
            if (total > room) partial[c] = 1;
            streamed[c] = total - at;
            const int64_t stored = h.host_slice_ptr[s1] - h.host_slice_ptr[s0];
            slow[c] = (int64_t)halo.size() > kHaloBase + kHaloPerColumn * stored;
            bytes[c] = fixed_bytes + (int)at * kColumnBytes;
        }
    });
    plan.faster = true;
    int64_t from_l2 = 0;
    for (int c = 0; c < grid; ++c) {
        if (!fits[c]) return;
        if (slow[c]) plan.faster = false;
        from_l2 += streamed[c] * kColumnBytes;
        plan.halo_ptr[c + 1] = plan.halo_ptr[c] + (int)halos[c].size();
        plan.smem = std::max(plan.smem, (size_t)bytes[c]);
        plan.hybrid = plan.hybrid || partial[c];
    }
    if ((double)from_l2 > kL2Share * (double)l2_bytes) plan.faster = false;
    plan.halo.reserve(plan.halo_ptr[grid]);
    for (auto& v : halos) plan.halo.insert(plan.halo.end(), v.begin(), v.end());
    plan.threads = 32 * warps;
    plan.grid = grid;
}

// Whether every CTA of the plan is resident at once.
cudaError_t onchip_allow(const OnchipPlan& plan, int sms, bool* resident) {
    const void* k = (const void*)oc_kernel(plan.meet, plan.threads, plan.hybrid != 0);
    cudaError_t err = allow_dynamic_smem(k, plan.smem);
    *resident = true;
    if (err != cudaSuccess || plan.meet == kAlone) return err;
    if (plan.meet == kCluster) {
        err = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (err != cudaSuccess) return err;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(plan.grid);
        cfg.blockDim = dim3(plan.threads);
        cfg.dynamicSmemBytes = plan.smem;
        cudaLaunchAttribute attr = cluster_attribute(plan.grid);
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        err = cudaOccupancyMaxActiveClusters(&clusters, k, &cfg);
        *resident = clusters > 0;
        return err;
    }
    int per_sm = 0;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, plan.threads, plan.smem);
    *resident = per_sm * sms >= plan.grid;
    return err;
}

cudaError_t launch_pcg_onchip(Handle& h, float dt, int write_state, float* q_out, float* v_out, float* f_ws,
                              cudaStream_t s, const float* solve_rhs, float* x_out, float tol, int maxiter,
                              bool solve_warm) {
    OcArgs a;
    a.valA = h.valA;
    a.valB = h.valB;
    a.valC = h.valC;
    a.lcol = h.oc_lcol;
    a.slice_ptr = h.slice_ptr;
    a.slice_meta = h.slice_meta;
    a.row_info = h.row_info;
    a.minv = h.minv;
    a.slice0 = h.oc_slice0;
    a.team = h.oc_team;
    a.kres = h.oc_kres;
    a.halo_ptr = h.oc_halo_ptr;
    a.halo = h.oc_halo;
    a.v4 = h.v4;
    a.q4 = h.q4;
    a.x4 = h.x;
    a.rest = h.rest;
    a.spring_ptr = h.node_spring_ptr;
    a.spring_ent = h.node_spring_ent;
    a.spring_idx = h.spring_idx;
    a.spring_kd = h.spring_kd;
    a.f_ws = f_ws;
    a.dv = x_out != nullptr ? x_out : h.dv;
    a.q_out = q_out;
    a.v_out = v_out;
    a.rec0 = h.oc_rec0;
    a.rec1 = h.oc_rec1;
    a.part = h.oc_part;
    a.barrier = h.oc_barrier;
    a.status = h.status;
    a.scene_stats = h.scene_stats;
    a.cum_iters = h.cum_iters;
    a.resid_max = h.resid_max;
    a.maxiter = maxiter >= 0 ? maxiter : h.maxiter;
    a.tol = tol > 0.0f ? tol : h.tol;
    a.dt = dt;
    a.limit_ns = h.wait_limit_ns;
    a.write_state = write_state;
    a.solve_rhs = solve_rhs;
    a.solve_warm = solve_warm ? 1 : 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(h.oc_grid);
    cfg.blockDim = dim3(h.oc_threads);
    cfg.dynamicSmemBytes = h.oc_smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    if (h.oc_meet == kCluster) {
        attr[1] = cluster_attribute(h.oc_grid);
    } else {
        attr[1].id = cudaLaunchAttributeCooperative;
        attr[1].val.cooperative = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = h.oc_meet == kAlone ? 1 : 2;  // one CTA waits for no other
    return cudaLaunchKernelEx(&cfg, oc_kernel(h.oc_meet, h.oc_threads, h.oc_hybrid != 0), a);
}

}  // namespace fem
