// nbh_force.cu — the force stage: Barnes-Hut tree walk with a group-voted opening test.
#include "nbh_common.cuh"
#include "nbh_kernels.h"

namespace nbh {

// Launch geometry is chosen at run time (nbh_autotune): threads per block (64 / 128 / 256)
// and the entries of each group's shared-memory stack.  A group whose stack would overflow
// restarts on the per-level (cell, next child) walk.
constexpr int kForceThreadsMax = 256;
constexpr int kStackCapMax = 256;
constexpr int kStackCapMin = 64;     // the deep walk keeps 2 * kMaxDepth ints in the same space

// The list walk (64-wide groups): per group, the records of accepted nodes awaiting
// evaluation (at most 31 wait after an evaluation and one round adds at most 32; separate
// arrays of x, y, z, m) with each record's full cell width^2 (for the error bound; 0 for a
// body), the undecided cells of a round (at most 32, likewise as arrays), the group's box and
// representatives, and a stack of `cap` cells whose children are still to be tested, with their
// level factors (a 64-entry stack also holds the per-level walk's 2 * kMaxDepth ints).
constexpr int kListCap = 64;
constexpr size_t list_group_bytes(int cap) {
    return kListCap * (sizeof(float4) + sizeof(float)) + 32 * sizeof(float4) + 4 * sizeof(float4) +
           (size_t)cap * sizeof(int2);
}
constexpr size_t force_list_smem_bytes(int threads, int cap) { return (size_t)(threads / 32) * list_group_bytes(cap); }

// Groups shared among the warps of a block: cells waiting per warp when they are dealt out, the
// room for the breadth-first queue, and what the warps tell each other.
constexpr int kSplitFront = 8;
constexpr int kSplitQueue = 256;
constexpr int kSplitMin = 4, kSplitMax = 8;
constexpr int kSplitKeep = kSplitQueue / (kSplitMin * 32);   // entries per lane of a warp's share, at most
struct SplitTeam {
    int item, status;
    int accepted[kSplitMax], opened[kSplitMax];
};
// Warps per group for `groups` groups.  Force stage of Plummer spheres in groups of 64, us, by the number
// of groups: 469 (30,000 bodies) 182 / 211 / 240 with 8 / 4 / 2 warps; 907 281 / 264 / 299; 1,250 383 /
// 297 / 311; 1,813 545 / 403 / 430; with 2 / 1 warps 1,875 465 / 385, 2,500 463 / 479, 3,125 571 / 563,
// 3,438 767 / 608: from 12 groups per SM on the warps' common first rounds cost more than idle schedulers
// do, and two warps are the best choice nowhere (in groups of 32 likewise: 1,032 groups 186 / 162 /
// 160, 1,782 291 / 217 / 283, 2 / 1 warps 1,875 315 / 225; of 128: 1,797 1208 / 848 / 913, 1,875 950 / 819,
// 3,594 1669 / 1171).  With kSplitFront 4 and 12 in place of 8: 172 and 149 us at 16,384 bodies (145),
// 262 and 306 at 65,536 (262).  The number of warps decides the order of a group's sum, so a
// universe's last bits depend on the batch it is in.
static int force_split(int groups, int sms) { return groups >= 12 * sms ? 1 : (groups >= 6 * sms ? 4 : 8); }
static_assert(kStackCapMin * sizeof(int2) >= 2 * kMaxDepth * sizeof(int), "the per-level walk fits the cell stack");

// The ordered walk: per group, a stack of pending nodes (24 bytes for each of the `cap` entries
// asked for, at 16 bytes each; 160 entries at least: with 96, 73 % of the groups of a 3M disc
// overflowed theirs, and walking them twice took 27115 us where the per-level walk alone takes
// 17143; with 160 12718), with their widths^2 factors where error bounds are recorded,
// the list of accepted records (each twice over where a lane has two or more bodies) with their
// widths^2, the undecided cells of a round, and the group's box and representatives.
constexpr int kOrderedMin = 160;
__host__ __device__ constexpr int ordered_entries(int cap) {
    return cap + cap / 2 > kOrderedMin ? cap + cap / 2 : kOrderedMin;
}
template <int W>
constexpr size_t force_smem_bytes(int threads, int cap, bool feat) {
    return (size_t)(threads / 32) * ((size_t)ordered_entries(cap) * (sizeof(float4) + (feat ? sizeof(float) : 0)) +
                                     kListCap * ((W >= 64 ? 2 : 1) * sizeof(float4) + sizeof(float)) +
                                     32 * sizeof(float4) + 4 * sizeof(float4));
}
// Free entries below which the ordered walk opens one cell a round instead of four (4M disc: 32
// and 80 the same at 256 entries asked for, 12073 and 12750 us at 192).
constexpr int kOrderedSlack = 32;

// Opening threshold of tree level L (root = 0): r^2/theta^2 * 4^-L + eps^2
// (calculateforce.cl:52-67).  The walk carries s = 4^-L (exact powers of two) and forms
// t0*s + eps^2, which equals ldexp(t0, -2L) + eps^2 in the normal range; below it eps^2
// absorbs the term either way.
__device__ __forceinline__ float level_dq(float t0, int level, float eps2) {
    return __fadd_rn(ldexpf(t0, -2 * level), eps2);
}

// 1/sqrt(d2).  d2 >= eps^2 > 0 is never subnormal, so the flush-to-zero form of the
// hardware approximation returns exactly what rsqrtf would.
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// max(a, b, 0), NaN if one of them is.  The centre of a cell of massless bodies is not a number
// (0 / 0) and passes no body's distance test; fmaxf would drop it and leave a distance of zero to
// the group's box.
__device__ __forceinline__ float gap_nan(float a, float b) {
    float y;
    asm("max.NaN.f32 %0, %1, %2, 0f00000000;" : "=f"(y) : "f"(a), "f"(b));
    return y;
}

// One accepted interaction (calculateforce.cl:146-151).  With FEAT it also accumulates
// the quadrupole error bound m s^2 / d^4 of an accepted cell of full width^2 s2 (0 for a
// body), the feature the learned opening angle is predicted from.
template <bool REF, bool FEAT>
__device__ __forceinline__ void interact(const float4 q, const float dx, const float dy, const float dz,
                                         const float d2, float& ax, float& ay, float& az, float& eb,
                                         const float s2) {
    float rd;
    if constexpr (REF) rd = __frcp_rn(__fsqrt_rn(d2));
    else rd = rsqrt_ftz(d2);
    const float f = __fmul_rn(__fmul_rn(__fmul_rn(q.w, rd), rd), rd);
    ax = madd<REF>(dx, f, ax);
    ay = madd<REF>(dy, f, ay);
    az = madd<REF>(dz, f, az);
    if constexpr (FEAT) eb = __fmaf_rn(__fmul_rn(f, rd), s2, eb);
}

template <bool REF>
__device__ __forceinline__ float dist2(const float dx, const float dy, const float dz, const float eps2) {
    if constexpr (REF)
        return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)), eps2);
    else
        return __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmaf_rn(dz, dz, eps2)));
}

// The list walk's arithmetic is packed: one FP32x2 instruction works on two consecutive records
// of the list.  FP32x2 has the multiply-add rate of scalar FP32 (measured 2.03-2.1 cycles per
// warp and scheduler against 2 x 1.11) but takes half the issue slots, and a list kept as
// separate arrays of x, y, z and m hands its operand pairs over straight from 16-byte shared
// loads, four records each, without a move.  A body's negated coordinates are held twice
// over, and its sums as one partial sum over the even and one over the odd records.  A 32-record
// batch for two bodies per lane, alone on an SM: 30.5 cycles per record and warp, 33.5 with
// scalar arithmetic and 16-byte records, and 15 issue slots per record instead of 27, which
// is what the walk's other instructions need.
struct ListBody {
    float2 nx, ny, nz;
};
struct ListSum {
    float2 x, y, z, e;
};

template <bool FEAT>
__device__ __forceinline__ void interact2(const float2 X, const float2 Y, const float2 Z, const float2 M,
                                          const float2 S, const ListBody& b, const float2 eps2, ListSum& a) {
    const float2 dx = __fadd2_rn(X, b.nx), dy = __fadd2_rn(Y, b.ny), dz = __fadd2_rn(Z, b.nz);
    const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, eps2)));
    const float2 rd = make_float2(rsqrt_ftz(d2.x), rsqrt_ftz(d2.y));
    const float2 f = __fmul2_rn(__fmul2_rn(__fmul2_rn(M, rd), rd), rd);
    a.x = __ffma2_rn(dx, f, a.x);
    a.y = __ffma2_rn(dy, f, a.y);
    a.z = __ffma2_rn(dz, f, a.z);
    if constexpr (FEAT) a.e = __ffma2_rn(__fmul2_rn(f, rd), S, a.e);
}

// Four records of the list (lst: arrays x, y, z, m and, with FEAT, width^2, kListCap apart;
// `at` a multiple of 4) for the lane's bodies.
template <int BPL, bool FEAT>
__device__ __forceinline__ void eval4(const float* lst, const int at, const ListBody (&b)[BPL], const float2 eps2,
                                      ListSum (&a)[BPL]) {
    const float4 X = *reinterpret_cast<const float4*>(lst + at);
    const float4 Y = *reinterpret_cast<const float4*>(lst + kListCap + at);
    const float4 Z = *reinterpret_cast<const float4*>(lst + 2 * kListCap + at);
    const float4 M = *reinterpret_cast<const float4*>(lst + 3 * kListCap + at);
    float4 S = make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (FEAT) S = *reinterpret_cast<const float4*>(lst + 4 * kListCap + at);
#pragma unroll
    for (int k = 0; k < BPL; ++k)
        interact2<FEAT>(make_float2(X.x, X.y), make_float2(Y.x, Y.y), make_float2(Z.x, Z.y), make_float2(M.x, M.y),
                        make_float2(S.x, S.y), b[k], eps2, a[k]);
#pragma unroll
    for (int k = 0; k < BPL; ++k)
        interact2<FEAT>(make_float2(X.z, X.w), make_float2(Y.z, Y.w), make_float2(Z.z, Z.w), make_float2(M.z, M.w),
                        make_float2(S.z, S.w), b[k], eps2, a[k]);
}

// The ordered walk's arithmetic: `cnt` records of the list from `at` on, each body's sums
// formed in list order.  Two or more bodies per lane (FMA arithmetic): FP32x2 over pairs of bodies,
// the records stored twice over as (x, x, y, y) and (z, z, m, m).  One body per lane: scalar.  16
// bodies on the warp's 32 lanes: the half-warps take one of two consecutive records each, and the
// lower half, which holds the sums, adds its own record's terms and then the other's.
template <int W, bool REF, bool FEAT>
__device__ __forceinline__ void eval_ordered(const float4* lst, const float* lw, const int at, const int cnt,
                                             const float4 (&pb)[W < 32 ? 1 : W / 32], const float eps2,
                                             float (&ax)[W < 32 ? 1 : W / 32], float (&ay)[W < 32 ? 1 : W / 32],
                                             float (&az)[W < 32 ? 1 : W / 32], float (&eb)[W < 32 ? 1 : W / 32]) {
    if constexpr (W >= 64) {
        static_assert(!REF, "two bodies per lane take FMA arithmetic");
        const float2 e2 = make_float2(eps2, eps2);
#pragma unroll 8
        for (int i = at; i < at + cnt; ++i) {
            const float4 xy = lst[2 * i], zm = lst[2 * i + 1];
            const float s2 = FEAT ? lw[i] : 0.0f;
#pragma unroll
            for (int k = 0; k < W / 32; k += 2) {
                const ListBody b = {make_float2(-pb[k].x, -pb[k + 1].x), make_float2(-pb[k].y, -pb[k + 1].y),
                                    make_float2(-pb[k].z, -pb[k + 1].z)};
                ListSum a = {make_float2(ax[k], ax[k + 1]), make_float2(ay[k], ay[k + 1]),
                             make_float2(az[k], az[k + 1]), make_float2(eb[k], eb[k + 1])};
                interact2<FEAT>(make_float2(xy.x, xy.y), make_float2(xy.z, xy.w), make_float2(zm.x, zm.y),
                                make_float2(zm.z, zm.w), make_float2(s2, s2), b, e2, a);
                ax[k] = a.x.x, ax[k + 1] = a.x.y, ay[k] = a.y.x, ay[k + 1] = a.y.y;
                az[k] = a.z.x, az[k + 1] = a.z.y;
                if constexpr (FEAT) eb[k] = a.e.x, eb[k + 1] = a.e.y;
            }
        }
    } else if constexpr (W == 32) {
#pragma unroll 4
        for (int i = at; i < at + cnt; ++i) {
            const float4 q = lst[i];
            const float dx = __fsub_rn(q.x, pb[0].x), dy = __fsub_rn(q.y, pb[0].y), dz = __fsub_rn(q.z, pb[0].z);
            interact<REF, FEAT>(q, dx, dy, dz, dist2<REF>(dx, dy, dz, eps2), ax[0], ay[0], az[0], eb[0],
                                FEAT ? lw[i] : 0.0f);
        }
    } else {
        const int half = (threadIdx.x >> 4) & 1;
#pragma unroll 4
        for (int i = 0; i < cnt; i += 2) {
            // (the record past an odd last one is whatever lies there; its terms are not added)
            const int r = (at + i + half) & (kListCap - 1);
            const float4 q = lst[r];
            const float dx = __fsub_rn(q.x, pb[0].x), dy = __fsub_rn(q.y, pb[0].y), dz = __fsub_rn(q.z, pb[0].z);
            const float d2 = dist2<REF>(dx, dy, dz, eps2);
            float rd;
            if constexpr (REF) rd = __frcp_rn(__fsqrt_rn(d2));
            else rd = rsqrt_ftz(d2);
            const float f = __fmul_rn(__fmul_rn(__fmul_rn(q.w, rd), rd), rd);
            ax[0] = madd<REF>(dx, f, ax[0]);
            ay[0] = madd<REF>(dy, f, ay[0]);
            az[0] = madd<REF>(dz, f, az[0]);
            float g = 0.0f, s2 = 0.0f;
            if constexpr (FEAT) {
                s2 = lw[r];
                g = __fmul_rn(f, rd);
                eb[0] = __fmaf_rn(g, s2, eb[0]);
            }
            const float f1 = __shfl_down_sync(0xffffffffu, f, 16);
            const float x1 = __shfl_down_sync(0xffffffffu, dx, 16), y1 = __shfl_down_sync(0xffffffffu, dy, 16),
                        z1 = __shfl_down_sync(0xffffffffu, dz, 16);
            float g1 = 0.0f, s1 = 0.0f;
            if constexpr (FEAT) {
                g1 = __shfl_down_sync(0xffffffffu, g, 16);
                s1 = __shfl_down_sync(0xffffffffu, s2, 16);
            }
            if (i + 1 < cnt) {
                ax[0] = madd<REF>(x1, f1, ax[0]);
                ay[0] = madd<REF>(y1, f1, ay[0]);
                az[0] = madd<REF>(z1, f1, az[0]);
                if constexpr (FEAT) eb[0] = __fmaf_rn(g1, s1, eb[0]);
            }
        }
    }
}

// -------------------------------------------------------------------------------------
// Force (calculateforce.cl:52-185).  A group of W bodies (W = 16: the reference's work-group,
// :99,145; W = 32, 64, 128: one, two, four bodies per lane) is W consecutive bodies of the
// depth-first order, and one warp walks its universe's tree.  A body child is always accepted; a
// cell child only if every body of the group sees d^2 + eps^2 >= dq[level] (work_group_all,
// :145), else it is opened.  Every lane of a group accepts the same children, so the group's
// interactions are counted once.  Lanes past the end of a universe walk with their group's
// first body, and for W = 16 the upper half-warp holds the same bodies as the lower, so no
// vote needs a predicate.  Work items (32 bodies; 64 and 128 for those widths) are handed out
// dynamically.  After the walk: the leapfrog velocity correction for step > 0 (:174-181) and the
// acceleration store (:183-185).
//
// REF: reference arithmetic (rounded products, 1/sqrt correctly rounded); otherwise FMA and
// the hardware inverse square root.  PB: per-body opening angle from theta_body (with
// p.theta_group, the smallest angle of the group for all its bodies).  FEAT:
// also accumulate each body's quadrupole error bound into acc.w.  With p.probe set the
// results go to p.probe (x, y, z, bound) and no body state changes (force probe).  With
// p.feat_gate set, a launch that does not match the step's place in the learned-theta
// schedule returns at once (the step graph holds a recording and a plain launch).
//
// The votes are taken lane-parallel, one child per lane: a body is accepted; a cell is accepted
// when even the group's bounding box passes the test (the box's distance components bound every
// body's from below, and the rounded subtractions, products or fused squares, sums and the
// comparison are monotone, so every body's own test passes), and opened when the group's body
// nearest the box centre fails it (then the vote fails; with per-body angles also when the body
// with the smallest angle fails it).  Only the remaining cells take the vote of every body, two
// cells after two.  Accepted records go to a list in shared memory, evaluated 32 at a time in a
// loop of arithmetic alone.
//
// The ordered walk (LIST = false) keeps the reference's order of accumulation (depth-first,
// children in order): its stack holds every pending node with its record, the next one in order
// on top: the record of an accepted node, or the index of a cell to open.  A round looks at the
// top 32, moves the accepted ones above the first cell to open to the list, decides the children
// of the first four cells to open, and puts them in those cells' places, the accepted nodes
// between them moving up.  Force stage against visiting one node at a time with a vote each, us:
// 4M disc (W = 64) 11928 / 13747, 1M Plummer sphere 2748 / 3178 (W = 32: 3046 / 3757); reference
// arithmetic at theta^2 1.5 with W = 16: 100,003 bodies 174 / 276, 1M 1378 / 2065 (one warp per
// group of 16 in place of two groups in the halves of a warp, which ran one after the other),
// with W = 32 182 / 231 and 1030 / 1021.
//
// LIST (W = 32, 64 or 128; FMA arithmetic): each round takes the children of up to four cells
// from a stack of cells alone; the records are accumulated in list order (rounding may differ
// from the ordered walk in the last bits).
//
// In both, a stack that would overflow restarts the group on the per-level walk (stack_cap
// entries: 256 by default; the 64-body groups of the benchmarked spheres need at most 99 in the
// list walk).
//
// SPLIT (with LIST): a block of S = 4 or 8 warps shares one group.  A group's walk is one
// chain of rounds, and a universe with fewer groups than the GPU has room for warps leaves
// most of it idle (16,384 bodies in groups of 32: 512 warps on 608 schedulers).  Every warp
// expands the tree from the root breadth first, all of them the same way, until kSplitFront
// cells per warp wait; then warp w keeps every S-th of them and walks on alone, and the sums are
// added in the order of the warps at the end.  The records accepted on the way are dealt out
// the same way.  S depends on the number of groups only (force_split), so that the launch
// geometry does not change the order of the sums; the number of universes beside one does.
template <int W, bool REF, bool PB, bool FEAT, bool LIST = false, bool SPLIT = false>
__device__ __forceinline__ void force_walk(const StepParams& p) {
    static_assert(!LIST || (W >= 32 && !REF), "the list walk takes whole-warp groups and FMA arithmetic");
    static_assert(!SPLIT || LIST, "only the list walk shares a group among warps");
    __shared__ SplitTeam team;
    const int wt = SPLIT ? (int)(threadIdx.x >> 5) : 0;   // this warp of the S that share a group
    const int S = SPLIT ? (int)(blockDim.x >> 5) : 1;
    if constexpr (SPLIT) {
        // one read of the status word for the whole block, which meets at barriers
        if (threadIdx.x == 0) team.status = load_status(p.st);
        __syncthreads();
        if (team.status) return;
    } else {
        if (load_status(p.st)) return;
    }
    if (p.feat_gate && theta_bound_step(p.st, p.st->step) != (p.feat_gate == 1)) return;
    constexpr int BPL = W < 32 ? 1 : W / 32;        // bodies per lane
    const int cap = p.stack_cap;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    const int grp = threadIdx.x >> 5;
    // ordered walk
    constexpr int kDup = BPL >= 2 ? 2 : 1;           // float4 per list record
    const int ocap = ordered_entries(cap);
    float4* const sq = reinterpret_cast<float4*>(smem_raw + grp * force_smem_bytes<W>(32, cap, FEAT));   // pending nodes
    float4* const ol = sq + ocap;
    float4* const ogc = ol + kDup * kListCap;
    float* const oud = reinterpret_cast<float*>(ogc + 4);
    float* const olw = oud + 4 * 32;
    float* const ssl = olw + kListCap;               // FEAT: level factor of each pending node (0: a body)
    // list walk: the group's list of accepted records and its stack of (cell, level)
    float* const lst = reinterpret_cast<float*>(smem_raw + (size_t)grp * list_group_bytes(SPLIT ? max(cap, kSplitQueue) : cap));
    float* const ud = LIST ? lst + 5 * kListCap : oud;   // undecided cells of a round: x, y, z, threshold
    float4* const gc = LIST ? reinterpret_cast<float4*>(ud + 4 * 32) : ogc;   // the group's box and representatives
    int2* const cst = reinterpret_cast<int2*>(gc + 4);
    // deep-tree walk: (cell, next) per level
    int* const snode = LIST ? reinterpret_cast<int*>(cst) : reinterpret_cast<int*>(sq);
    int* const snext = snode + kMaxDepth;
    const int nbody = p.nbody;
    const float eps2 = p.eps2;
    const int step = p.st->step;
    const float4* __restrict__ node4 = p.node4;
    const int* __restrict__ child = p.child;
    const float4* __restrict__ kids4 = p.kids4;
    const int2* __restrict__ items = BPL == 4 ? p.items128 : (BPL == 2 ? p.items64 : p.warps);
    // 32-body items are two groups of 16
    const int nitems = BPL == 4 ? p.nitems128 : (BPL == 2 ? p.nitems64 : (W < 32 ? 2 * p.nwarps : p.nwarps));
    unsigned long long my_inter = 0;

    for (;;) {
        int item = 0;
        if constexpr (SPLIT) {
            __syncthreads();                 // the last group's sums have been read
            if (threadIdx.x == 0) team.item = atomicAdd(&p.st->force_next, 1);
            __syncthreads();
            item = team.item;
        } else {
            if (lane == 0) item = atomicAdd(&p.st->force_next, 1);
            item = __shfl_sync(0xffffffffu, item, 0);
        }
        if (item >= nitems) break;
        const int half = W < 32 ? item & 1 : 0;
        if (W < 32) item >>= 1;
        if (p.item_order) item = p.item_order[item];   // costly items first (see order_items)
        const int2 wi = items[item];
        const int u = wi.y;
        const int uend = p.ubody[u + 1];
        const int gfirst = wi.x + 16 * half;
        if (W < 32 && gfirst >= uend) continue;         // the item's second group has no bodies
        const float r = p.uradius[u];
        const float rr = __fmul_rn(r, r);
        float4 pb[BPL];
        float t0[BPL];
        float ax[BPL], ay[BPL], az[BPL], eb[BPL];
#pragma unroll
        for (int k = 0; k < BPL; ++k) {
            // lanes past the universe's end take their group's first body
            const int sk = gfirst + 32 * k + (W < 32 ? lane & 15 : lane);
            const int bk = p.sorted[sk < uend ? sk : gfirst];
            pb[k] = node4[bk];
            float th2 = p.theta2;
            if constexpr (PB) {
                const float th = p.theta_body[bk];
                th2 = __fmul_rn(th, th);
            }
            t0[k] = th2 > 0.0f ? __fdiv_rn(rr, th2) : rr;
            ax[k] = ay[k] = az[k] = eb[k] = 0.f;
        }
        if constexpr (PB) {
            if (p.theta_group) {
                // the group walks with its smallest angle (largest r^2 / theta^2), the walk
                // of a fixed angle; lanes past the end hold the first body's angle
                float tm = t0[0];
#pragma unroll
                for (int k = 1; k < BPL; ++k) tm = fmaxf(tm, t0[k]);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, o));
#pragma unroll
                for (int k = 0; k < BPL; ++k) t0[k] = tm;
            }
        }
        long long ninter = 0;
        int visits = 0;                                 // cost of this group's walk
        const int root = p.nnodes - u;

        {
            bool walked = true;
            {
                // the group's bounding box (lanes past the end hold the first body)
                float lox = pb[0].x, loy = pb[0].y, loz = pb[0].z, hix = pb[0].x, hiy = pb[0].y, hiz = pb[0].z;
#pragma unroll
                for (int k = 1; k < BPL; ++k) {
                    lox = fminf(lox, pb[k].x), loy = fminf(loy, pb[k].y), loz = fminf(loz, pb[k].z);
                    hix = fmaxf(hix, pb[k].x), hiy = fmaxf(hiy, pb[k].y), hiz = fmaxf(hiz, pb[k].z);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    lox = fminf(lox, __shfl_xor_sync(0xffffffffu, lox, o));
                    loy = fminf(loy, __shfl_xor_sync(0xffffffffu, loy, o));
                    loz = fminf(loz, __shfl_xor_sync(0xffffffffu, loz, o));
                    hix = fmaxf(hix, __shfl_xor_sync(0xffffffffu, hix, o));
                    hiy = fmaxf(hiy, __shfl_xor_sync(0xffffffffu, hiy, o));
                    hiz = fmaxf(hiz, __shfl_xor_sync(0xffffffffu, hiz, o));
                }
                // the representative: the body nearest the box centre (lowest index on ties)
                const float cx = 0.5f * (lox + hix), cy = 0.5f * (loy + hiy), cz = 0.5f * (loz + hiz);
                float best = 0.0f;
                int bid = 0;
#pragma unroll
                for (int k = 0; k < BPL; ++k) {
                    const float ex = pb[k].x - cx, ey = pb[k].y - cy, ez = pb[k].z - cz;
                    const float d = ex * ex + ey * ey + ez * ez;
                    if (k == 0 || d < best) {
                        best = d;
                        bid = lane * BPL + k;
                    }
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const float ob = __shfl_xor_sync(0xffffffffu, best, o);
                    const int oi = __shfl_xor_sync(0xffffffffu, bid, o);
                    if (ob < best || (ob == best && oi < bid)) {
                        best = ob;
                        bid = oi;
                    }
                }
                const int rsrc = bid / BPL, rk = bid % BPL;
                float4 rp = pb[0];
                float rt = t0[0];
#pragma unroll
                for (int k = 1; k < BPL; ++k)
                    if (rk == k) {
                        rp = pb[k];
                        rt = t0[k];
                    }
                rp.x = __shfl_sync(0xffffffffu, rp.x, rsrc);
                rp.y = __shfl_sync(0xffffffffu, rp.y, rsrc);
                rp.z = __shfl_sync(0xffffffffu, rp.z, rsrc);
                // thresholds: the box takes the group's largest r^2/theta^2 (the smallest angle)
                float tlb = t0[0], trep = t0[0];
                if constexpr (PB) {
#pragma unroll
                    for (int k = 1; k < BPL; ++k) tlb = fmaxf(tlb, t0[k]);
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) tlb = fmaxf(tlb, __shfl_xor_sync(0xffffffffu, tlb, o));
                    trep = __shfl_sync(0xffffffffu, rt, rsrc);
                }
                // per-body angles: a second representative, the body with the smallest angle
                // (the largest r^2/theta^2, the box's threshold; lowest index on ties) -- a
                // vote fails most often on it (learned step 2.36 -> 2.32 ms at 1M)
                float4 rp2 = rp;
                if constexpr (PB) {
                    float bt = t0[0];
                    int bi = lane * BPL;
#pragma unroll
                    for (int k = 1; k < BPL; ++k)
                        if (t0[k] > bt) {
                            bt = t0[k];
                            bi = lane * BPL + k;
                        }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        const float ob = __shfl_xor_sync(0xffffffffu, bt, o);
                        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                        if (ob > bt || (ob == bt && oi < bi)) {
                            bt = ob;
                            bi = oi;
                        }
                    }
                    const int r2src = bi / BPL, r2k = bi % BPL;
                    float4 mine2 = pb[0];
#pragma unroll
                    for (int k = 1; k < BPL; ++k)
                        if (r2k == k) mine2 = pb[k];
                    rp2.x = __shfl_sync(0xffffffffu, mine2.x, r2src);
                    rp2.y = __shfl_sync(0xffffffffu, mine2.y, r2src);
                    rp2.z = __shfl_sync(0xffffffffu, mine2.z, r2src);
                }
                if (lane == 0) {
                    gc[0] = make_float4(lox, loy, loz, tlb);
                    gc[1] = make_float4(hix, hiy, hiz, trep);
                    gc[2] = rp;
                    if constexpr (PB) gc[3] = rp2;
                }
            }
            const unsigned lt = (1u << lane) - 1u;
            if constexpr (LIST) {
                // from here on the bodies are held as ListBody (the empty asm keeps the compiler
                // from holding their plain coordinates beside it)
                ListBody lb[BPL];
                ListSum ls[BPL];
#pragma unroll
                for (int k = 0; k < BPL; ++k) {
                    float nx = -pb[k].x, ny = -pb[k].y, nz = -pb[k].z;
                    asm volatile("" : "+f"(nx), "+f"(ny), "+f"(nz));
                    lb[k].nx = make_float2(nx, nx), lb[k].ny = make_float2(ny, ny), lb[k].nz = make_float2(nz, nz);
                    ls[k].x = ls[k].y = ls[k].z = ls[k].e = make_float2(0.f, 0.f);
                }
                const float2 eps22 = make_float2(eps2, eps2);
                if (lane == 0) cst[0] = make_int2(root, __float_as_int(1.0f));
                int ctop = 1, opened = 0;              // every tested child is accepted or opened
                // breadth first (SPLIT) until there are enough cells to share: the cells from
                // `head` on wait in order; dealt: accepted records so far
                bool spread = SPLIT;
                int head = 0, dealt = 0;
                // the list is a ring of kListCap records; the first of the lcnt waiting ones is at
                // lbase, 0 or 32
                int lcnt = 0, lbase = 0;
                int accepted = 0;                      // one body's: below the body count
                __syncwarp();
                for (;;) {
                    if (SPLIT && spread &&
                        (ctop == head || ctop - head >= kSplitFront * S || ctop + 32 > kSplitQueue)) {
                        // this warp's share, moved to the bottom
                        int2 keep[kSplitKeep];
#pragma unroll
                        for (int k = 0; k < kSplitKeep; ++k) {
                            const int at = head + wt + S * (lane + 32 * k);
                            keep[k] = at < ctop ? cst[at] : make_int2(kNull, 0);
                        }
                        __syncwarp();
                        const int mine = (ctop - head - wt + S - 1) / S;
#pragma unroll
                        for (int k = 0; k < kSplitKeep; ++k)
                            if (keep[k].x != kNull) cst[lane + 32 * k] = keep[k];
                        ctop = max(mine, 0);
                        spread = false;
                        __syncwarp();
                    }
                    if (ctop == 0) break;
                    const int k4 = min(4, spread ? ctop - head : ctop);
                    const int ci = lane >> 3;
                    int chk = kNull;
                    float sl = 1.0f;                    // 4^-level of the cell whose child this is
                    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (ci < k4) {
                        const int2 e = cst[spread ? head + ci : ctop - 1 - ci];
                        sl = __int_as_float(e.y);
                        const size_t o8 = ((size_t)(e.x - nbody) << 3) + (lane & 7);
                        chk = __ldg(child + o8);
                        q = __ldg(kids4 + o8);
                    }
                    if (spread) head += k4;
                    else ctop -= k4;
                    __syncwarp();          // the popped entries are read before pushes reuse them
                    // children of a level-lv cell: t0 * 4^-lv + eps^2 (4^-lv exact)
                    bool acc = chk >= 0 && chk < nbody;
                    bool opn = false, inc = false;
                    float qlb = 0.0f;
                    if (chk >= nbody) {
                        const float4 lo = gc[0], hi = gc[1];
                        const float gx = gap_nan(__fsub_rn(q.x, hi.x), __fsub_rn(lo.x, q.x));
                        const float gy = gap_nan(__fsub_rn(q.y, hi.y), __fsub_rn(lo.y, q.y));
                        const float gz = gap_nan(__fsub_rn(q.z, hi.z), __fsub_rn(lo.z, q.z));
                        const float dlb = dist2<false>(gx, gy, gz, eps2);
                        qlb = PB ? __fmaf_rn(lo.w, sl, eps2) : __fadd_rn(__fmul_rn(lo.w, sl), eps2);
                        if (dlb >= qlb) {
                            acc = true;
                        } else {
                            const float4 r1 = gc[2];
                            const float rx = __fsub_rn(q.x, r1.x), ry = __fsub_rn(q.y, r1.y), rz = __fsub_rn(q.z, r1.z);
                            const float qr = PB ? __fmaf_rn(hi.w, sl, eps2) : qlb;
                            if (dist2<false>(rx, ry, rz, eps2) < qr) {
                                opn = true;
                            } else if constexpr (PB) {
                                // the smallest-angle body's own test (its threshold is the box's)
                                const float4 r2 = gc[3];
                                const float sx = __fsub_rn(q.x, r2.x), sy = __fsub_rn(q.y, r2.y),
                                            sz = __fsub_rn(q.z, r2.z);
                                if (dist2<false>(sx, sy, sz, eps2) < qlb) opn = true;
                                else inc = true;
                            } else {
                                inc = true;
                            }
                        }
                    }
                    // undecided cells: the vote of every body, two cells after two
                    const unsigned im = __ballot_sync(0xffffffffu, inc);
                    if (im) {
                        // their records go to shared memory and every lane reads them back in turn,
                        // with the finished threshold (fixed angle) or the level factor; the second
                        // cell of an odd last pair is whatever lies there, its vote is not used
                        const int nud = __popc(im);
                        const int mine = __popc(im & lt);
                        if (inc) {
                            ud[mine] = q.x;
                            ud[32 + mine] = q.y;
                            ud[64 + mine] = q.z;
                            ud[96 + mine] = PB ? sl : qlb;
                        }
                        __syncwarp();
                        unsigned res = 0;
                        for (int j = 0; j < nud; j += 2) {
                            const float2 ux = *reinterpret_cast<const float2*>(ud + j);
                            const float2 uy = *reinterpret_cast<const float2*>(ud + 32 + j);
                            const float2 uz = *reinterpret_cast<const float2*>(ud + 64 + j);
                            const float2 uq = *reinterpret_cast<const float2*>(ud + 96 + j);
                            bool pass0 = true, pass1 = true;
#pragma unroll
                            for (int k = 0; k < BPL; ++k) {
                                const float2 dx = __fadd2_rn(ux, lb[k].nx);
                                const float2 dy = __fadd2_rn(uy, lb[k].ny);
                                const float2 dz = __fadd2_rn(uz, lb[k].nz);
                                const float2 d2 =
                                    __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, eps22)));
                                pass0 = pass0 && d2.x >= (PB ? __fmaf_rn(t0[k], uq.x, eps2) : uq.x);
                                pass1 = pass1 && d2.y >= (PB ? __fmaf_rn(t0[k], uq.y, eps2) : uq.y);
                            }
                            res |= (__all_sync(0xffffffffu, pass0) ? 1u : 0u) << j;
                            res |= (__all_sync(0xffffffffu, pass1) ? 2u : 0u) << j;
                        }
                        if (inc) {
                            acc = (res >> mine) & 1u;
                            opn = !acc;
                        }
                    }
                    const unsigned om = __ballot_sync(0xffffffffu, opn);
                    const int on = __popc(om);
                    if (SPLIT && spread) {
                        const unsigned every = __ballot_sync(0xffffffffu, acc);
                        acc = acc && ((dealt + __popc(every & lt)) & (S - 1)) == wt;
                        dealt += __popc(every);
                        if (wt == 0) opened += on;
                    } else {
                        opened += on;
                        if (ctop + on > cap) {           // group-uniform
                            walked = false;
                            break;
                        }
                    }
                    const unsigned am = __ballot_sync(0xffffffffu, acc);
                    if (acc) {
                        const int at = (lbase + lcnt + __popc(am & lt)) & (kListCap - 1);
                        lst[at] = q.x;
                        lst[kListCap + at] = q.y;
                        lst[2 * kListCap + at] = q.z;
                        lst[3 * kListCap + at] = q.w;
                        // full width^2 of an accepted cell, r^2 * 4^-level (0 for a body)
                        if constexpr (FEAT) lst[4 * kListCap + at] = chk >= nbody ? __fmul_rn(rr, sl) : 0.0f;
                    }
                    // children of a cell at level 63 are bodies: the factor stays a normal number
                    if (opn) cst[ctop + __popc(om & lt)] = make_int2(chk, __float_as_int(__fmul_rn(sl, 0.25f)));
                    lcnt += __popc(am);
                    ctop += on;
                    __syncwarp();          // list and stack written before they are read
                    if (lcnt >= 32) {
                        // 32 records at a time (two or more bodies per lane: unrolled completely, a 1M
                        // step 2433 us against 2526 unrolled by 2, 256 universes 5796 against 5980);
                        // at most 31 wait behind them
#pragma unroll(BPL >= 2 ? 8 : 2)
                        for (int i = 0; i < 32; i += 4) eval4<BPL, FEAT>(lst + lbase, i, lb, eps22, ls);
                        accepted += 32;
                        lcnt -= 32;
                        lbase ^= 32;
                    }
                }
                if (walked) {
                    if (lcnt > 0) {
                        // the last records, filled up to a multiple of four with massless ones
                        if (lane < (-lcnt & 3)) {
                            const int at = lbase + lcnt + lane;
#pragma unroll
                            for (int f = 0; f < (FEAT ? 5 : 4); ++f) lst[f * kListCap + at] = 0.0f;
                        }
                        __syncwarp();
                        for (int i = 0; i < lcnt; i += 4) eval4<BPL, FEAT>(lst + lbase, i, lb, eps22, ls);
                        accepted += lcnt;
                        __syncwarp();
                    }
#pragma unroll
                    for (int k = 0; k < BPL; ++k) {
                        ax[k] = __fadd_rn(ls[k].x.x, ls[k].x.y);
                        ay[k] = __fadd_rn(ls[k].y.x, ls[k].y.y);
                        az[k] = __fadd_rn(ls[k].z.x, ls[k].z.y);
                        if constexpr (FEAT) eb[k] = __fadd_rn(ls[k].e.x, ls[k].e.y);
                    }
                }
                if constexpr (SPLIT) {
                    // the warps' sums through shared memory (each in its own list's place, which every
                    // lane has finished reading)
                    __syncwarp();
                    float4* const out = reinterpret_cast<float4*>(lst);
#pragma unroll
                    for (int k = 0; k < BPL; ++k) out[32 * k + lane] = make_float4(ax[k], ay[k], az[k], eb[k]);
                    if (lane == 0) team.accepted[wt] = walked ? accepted : -1, team.opened[wt] = opened;
                    __syncthreads();
                    if (wt != 0) continue;               // the first warp finishes the group
                    for (int w = 1; w < S; ++w) {
                        const float4* const from = reinterpret_cast<const float4*>(
                            smem_raw + (size_t)w * list_group_bytes(max(cap, kSplitQueue)));
                        if (team.accepted[w] < 0) walked = false;
                        accepted += team.accepted[w];
                        opened += team.opened[w];
#pragma unroll
                        for (int k = 0; k < BPL; ++k) {
                            const float4 f = from[32 * k + lane];
                            ax[k] = __fadd_rn(ax[k], f.x);
                            ay[k] = __fadd_rn(ay[k], f.y);
                            az[k] = __fadd_rn(az[k], f.z);
                            if constexpr (FEAT) eb[k] = __fadd_rn(eb[k], f.w);
                        }
                    }
                }
                if (walked) {
                    ninter = accepted;
                    visits = accepted + opened;
                } else {
#pragma unroll
                    for (int k = 0; k < BPL; ++k) {
                        ax[k] = ay[k] = az[k] = eb[k] = 0.0f;
                        pb[k].x = -lb[k].nx.x, pb[k].y = -lb[k].ny.x, pb[k].z = -lb[k].nz.x;
                    }
                    __syncwarp();
                }
            } else {
                // a pending cell to open: its index, the level factor of its parent's children (the
                // root: 4, so that its own children's is 1), and kOpenTag in place of the mass
                constexpr int kOpenTag = -1;
                if (lane == 0)
                    sq[0] = make_float4(__int_as_float(root), 4.0f, 0.0f, __int_as_float(kOpenTag));
                int top = 1, opened = 0, accepted = 0;
                int lcnt = 0, lbase = 0;               // the list is a ring, as in the list walk
                __syncwarp();
                while (top > 0) {
                    const int T = min(32, top);
                    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                    float sl = 0.0f;
                    if (lane < T) {
                        q = sq[top - 1 - lane];
                        if constexpr (FEAT) sl = ssl[top - 1 - lane];
                    }
                    const bool opn = lane < T && __float_as_int(q.w) == kOpenTag;
                    const unsigned om = __ballot_sync(0xffffffffu, opn);
                    // accepted nodes above the first cell to open: next in order, to the list
                    const int emit = om ? __ffs((int)om) - 1 : T;
                    if (lane < emit) {
                        const int at = (lbase + lcnt + lane) & (kListCap - 1);
                        if constexpr (kDup == 2) {
                            ol[2 * at] = make_float4(q.x, q.x, q.y, q.y);
                            ol[2 * at + 1] = make_float4(q.z, q.z, q.w, q.w);
                        } else {
                            ol[at] = q;
                        }
                        if constexpr (FEAT) olw[at] = __fmul_rn(rr, sl);
                    }
                    lcnt += emit;
                    if (!om) {
                        top -= T;
                    } else {
                        // the first four cells to open, at most, at lanes at[0] < at[1] < ...
                        int at[4], last = emit;
                        unsigned m = om;
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            at[g] = m ? __ffs((int)m) - 1 : 32;
                            if (m) last = at[g];
                            m &= m - 1;
                        }
                        // one at a time when their children might not fit (group-uniform)
                        if (top - 1 - emit + 32 > ocap - kOrderedSlack) {
                            last = emit;
                            at[1] = at[2] = at[3] = 32;
                        }
                        const int g = lane >> 3;
                        const int from = g == 0 ? at[0] : (g == 1 ? at[1] : (g == 2 ? at[2] : at[3]));
                        const int cell = __float_as_int(__shfl_sync(0xffffffffu, q.x, from & 31));
                        const float csl = __fmul_rn(__shfl_sync(0xffffffffu, q.y, from & 31), 0.25f);
                        int ch = kNull;
                        float4 cq = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (from < 32) {
                            const size_t o8 = ((size_t)(cell - nbody) << 3) + (lane & 7);
                            ch = __ldg(child + o8);
                            cq = __ldg(kids4 + o8);
                        }
                        // the children's votes
                        bool keep = ch >= 0 && ch < nbody, inc = false;   // keep: accepted
                        float qlb = 0.0f;
                        if (ch >= nbody) {
                            const float4 lo = gc[0], hi = gc[1];
                            const float gx = gap_nan(__fsub_rn(cq.x, hi.x), __fsub_rn(lo.x, cq.x));
                            const float gy = gap_nan(__fsub_rn(cq.y, hi.y), __fsub_rn(lo.y, cq.y));
                            const float gz = gap_nan(__fsub_rn(cq.z, hi.z), __fsub_rn(lo.z, cq.z));
                            // t0 * 4^-level is exact, so the fused form gives the same threshold
                            qlb = __fmaf_rn(lo.w, csl, eps2);
                            if (dist2<REF>(gx, gy, gz, eps2) >= qlb) {
                                keep = true;
                            } else {
                                const float4 r1 = gc[2];
                                const float rx = __fsub_rn(cq.x, r1.x), ry = __fsub_rn(cq.y, r1.y),
                                            rz = __fsub_rn(cq.z, r1.z);
                                inc = !(dist2<REF>(rx, ry, rz, eps2) < (PB ? __fmaf_rn(hi.w, csl, eps2) : qlb));
                                if constexpr (PB) {
                                    const float4 r2 = gc[3];
                                    const float sx = __fsub_rn(cq.x, r2.x), sy = __fsub_rn(cq.y, r2.y),
                                                sz = __fsub_rn(cq.z, r2.z);
                                    inc = inc && !(dist2<REF>(sx, sy, sz, eps2) < qlb);
                                }
                            }
                        }
                        const unsigned im = __ballot_sync(0xffffffffu, inc);
                        if (im) {
                            const int nud = __popc(im);
                            const int mine = __popc(im & lt);
                            if (inc)
                                reinterpret_cast<float4*>(ud)[mine] = make_float4(cq.x, cq.y, cq.z, PB ? csl : qlb);
                            __syncwarp();
                            unsigned res = 0;
#pragma unroll 2
                            for (int j = 0; j < nud; ++j) {
                                const float4 uq = reinterpret_cast<const float4*>(ud)[j];
                                bool pass = true;
#pragma unroll
                                for (int k = 0; k < BPL; ++k) {
                                    const float dx = __fsub_rn(uq.x, pb[k].x), dy = __fsub_rn(uq.y, pb[k].y),
                                                dz = __fsub_rn(uq.z, pb[k].z);
                                    pass = pass && dist2<REF>(dx, dy, dz, eps2) >=
                                                       (PB ? __fmaf_rn(t0[k], uq.w, eps2) : uq.w);
                                }
                                res |= (__all_sync(0xffffffffu, pass) ? 1u : 0u) << j;
                            }
                            if (inc) keep = (res >> mine) & 1u;
                        }
                        const unsigned vm = __ballot_sync(0xffffffffu, ch >= 0);
                        const unsigned am = ~om & ~((1u << emit) - 1u) & ((1u << last) - 1u);   // moving up
                        const int n = __popc(am) + __popc(vm);
                        const int base = top - 1 - last;
                        if (base + n > ocap) {         // group-uniform
                            walked = false;
                            break;
                        }
                        opened += 1 + __popc(om & ((1u << last) - 1u));
                        __syncwarp();                  // the window has been read
                        if ((am >> lane) & 1u) {
                            int ord = __popc(am & lt);
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                if (at[k] < lane) ord += __popc((vm >> (8 * k)) & 0xffu);
                            sq[base + n - 1 - ord] = q;
                            if constexpr (FEAT) ssl[base + n - 1 - ord] = sl;
                        }
                        if (ch >= 0) {
                            const int ord = __popc(am & ((1u << from) - 1u)) + __popc(vm & lt);
                            sq[base + n - 1 - ord] =
                                keep ? cq : make_float4(__int_as_float(ch), csl, 0.0f, __int_as_float(kOpenTag));
                            if constexpr (FEAT) ssl[base + n - 1 - ord] = ch >= nbody ? csl : 0.0f;
                        }
                        top = base + n;
                    }
                    __syncwarp();
                    if (lcnt >= 32) {
                        eval_ordered<W, REF, FEAT>(ol, olw, lbase, 32, pb, eps2, ax, ay, az, eb);
                        accepted += 32;
                        lcnt -= 32;
                        lbase ^= 32;
                        __syncwarp();
                    }
                }
                if (walked) {
                    eval_ordered<W, REF, FEAT>(ol, olw, lbase, lcnt, pb, eps2, ax, ay, az, eb);
                    ninter = accepted + lcnt;
                    visits = accepted + lcnt + opened;
                } else {
#pragma unroll
                    for (int k = 0; k < BPL; ++k) ax[k] = ay[k] = az[k] = eb[k] = 0.0f;
                }
                __syncwarp();
            }
            if (!walked) {
                // The stack was full: per-level (cell, next child) walk (calculateforce.cl:112-172).
                if (lane == 0) atomicAdd(&p.st->restarts, 1);
                int depth = 0;
                int node = root;
                int k8 = 0;
                float dq[BPL];
#pragma unroll
                for (int k = 0; k < BPL; ++k) dq[k] = level_dq(t0[k], 0, eps2);
                for (;;) {
                    int ch = kNull;
                    if (k8 < 8) ch = __ldg(child + ((size_t)(node - nbody) << 3) + k8);
                    if (ch < 0) {
                        if (depth == 0) break;
                        --depth;
                        node = snode[depth];
                        k8 = snext[depth];
#pragma unroll
                        for (int k = 0; k < BPL; ++k) dq[k] = level_dq(t0[k], depth, eps2);
                        continue;
                    }
                    ++k8;
                    const float4 q = __ldg(node4 + ch);
                    float dx[BPL], dy[BPL], dz[BPL], d2[BPL];
                    bool pass = true;
#pragma unroll
                    for (int k = 0; k < BPL; ++k) {
                        dx[k] = __fsub_rn(q.x, pb[k].x);
                        dy[k] = __fsub_rn(q.y, pb[k].y);
                        dz[k] = __fsub_rn(q.z, pb[k].z);
                        d2[k] = dist2<REF>(dx[k], dy[k], dz[k], eps2);
                        pass = pass && d2[k] >= dq[k];
                    }
                    if (ch < nbody || __all_sync(0xffffffffu, pass)) {
                        const float s2 = ch >= nbody ? ldexpf(rr, -2 * depth) : 0.0f;
#pragma unroll
                        for (int k = 0; k < BPL; ++k)
                            interact<REF, FEAT>(q, dx[k], dy[k], dz[k], d2[k], ax[k], ay[k], az[k], eb[k], s2);
                        ++ninter;
                    } else {
                        if (depth + 1 >= kMaxDepth) {   // unreachable for a tree the build accepted
                            raise_error(p.st, NBH_ERR_DEPTH);
                            break;
                        }
                        // every lane writes the same entry, so no lane reads a stale one
                        snode[depth] = node;
                        snext[depth] = k8;
                        ++depth;
                        node = ch;
                        k8 = 0;
#pragma unroll
                        for (int k = 0; k < BPL; ++k) dq[k] = level_dq(t0[k], depth, eps2);
                    }
                }
            }
        }

#pragma unroll
        for (int k = 0; k < BPL; ++k) {
            // looked up again rather than held in registers through the walk
            const int sk = gfirst + 32 * k + lane;
            if (sk >= p.ubody[u + 1] || (W < 32 && lane >= W)) continue;
            const int bk = p.sorted[sk];
            if (p.G != 1.0f) {
                ax[k] = __fmul_rn(ax[k], p.G);
                ay[k] = __fmul_rn(ay[k], p.G);
                az[k] = __fmul_rn(az[k], p.G);
                eb[k] = __fmul_rn(eb[k], p.G);
            }
            my_inter += (unsigned long long)ninter;
            if (p.probe) {
                p.probe[bk] = make_float4(ax[k], ay[k], az[k], eb[k]);
                continue;
            }
            float4 v = p.vel[bk];
            const float4 ao = p.acc[bk];
            if (step > 0) {
                const float tx = __fmul_rn(__fsub_rn(ax[k], ao.x), p.dt);
                const float ty = __fmul_rn(__fsub_rn(ay[k], ao.y), p.dt);
                const float tz = __fmul_rn(__fsub_rn(az[k], ao.z), p.dt);
                if (p.precise) {
                    float4 kv = p.kvel[bk];
                    float y1, t1;
                    y1 = __fsub_rn(__fmul_rn(tx, 0.5f), kv.x); t1 = __fadd_rn(v.x, y1); kv.x = __fsub_rn(__fsub_rn(t1, v.x), y1); v.x = t1;
                    y1 = __fsub_rn(__fmul_rn(ty, 0.5f), kv.y); t1 = __fadd_rn(v.y, y1); kv.y = __fsub_rn(__fsub_rn(t1, v.y), y1); v.y = t1;
                    y1 = __fsub_rn(__fmul_rn(tz, 0.5f), kv.z); t1 = __fadd_rn(v.z, y1); kv.z = __fsub_rn(__fsub_rn(t1, v.z), y1); v.z = t1;
                    p.kvel[bk] = kv;
                } else {
                    v.x = madd<REF>(tx, 0.5f, v.x);
                    v.y = madd<REF>(ty, 0.5f, v.y);
                    v.z = madd<REF>(tz, 0.5f, v.z);
                }
                p.vel[bk] = v;
            }
            p.acc[bk] = make_float4(ax[k], ay[k], az[k], eb[k]);
        }
        if (p.item_cost) {
            // the item's cost: its group's visits (the deep walk counts accepted children), the
            // first of two groups' (W = 16)
            const int c = visits > 0 ? visits : (int)min(ninter, (long long)0x7fffffff);
            if (lane == 0 && half == 0) p.item_cost[item] = c;
        }
        __syncwarp();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) my_inter += __shfl_xor_sync(0xffffffffu, my_inter, o);
    if (lane == 0 && my_inter) atomicAdd(&p.st->interactions, my_inter);
}

// The kernels.  The 64-wide walks ask for resident blocks of the largest geometry, which
// bounds their registers: 3 (up to 80 registers) for all but the plain list walk, which fits in
// 64 without spills and takes 4 (measured, us per step with 4 against 3: 256-universe ensemble
// 6407 against 6488, 1M sphere 2618 against 2600; the list walk with per-body angles spills at
// 64: 8 learned steps 18143 against 17435).  The ordered
// walks take 79-80 (4M disc with 64 registers: 12291 against 11928).
// The other widths keep the compiler's own choice.
template <int W, bool REF, bool PB, bool FEAT, bool LIST = false>
__global__ void __launch_bounds__(kForceThreadsMax) force_kernel(StepParams p) {
    force_walk<W, REF, PB, FEAT, LIST>(p);
}
template <bool PB, bool FEAT, bool LIST>
__global__ void __launch_bounds__(kForceThreadsMax, LIST && !PB && !FEAT ? 4 : 3) force_kernel64(StepParams p) {
    force_walk<64, false, PB, FEAT, LIST>(p);
}

template <int W, bool PB, bool FEAT>
__global__ void __launch_bounds__(32 * kSplitMax) force_split_kernel(StepParams p) {
    force_walk<W, false, PB, FEAT, true, true>(p);
}

template <int W, bool REF, bool PB, bool FEAT, bool LIST = false>
static auto force_entry() {
    if constexpr (W == 64 && !REF) return force_kernel64<PB, FEAT, LIST>;
    else return force_kernel<W, REF, PB, FEAT, LIST>;
}

// -------------------------------------------------------------------------------------
template <int W, bool REF, bool PB>
static void launch_force_pf(const StepParams& p, bool feat, int grid, int threads, cudaStream_t s) {
    // No more blocks than there are groups for: with more, the SMs whose blocks start first take all
    // groups and others stay idle (64-wide, 240,000 bodies, 3,750 groups for room for 4,864: 745 us
    // against 610).
    const int groups = W == 128 ? p.nitems128 : (W == 64 ? p.nitems64 : (W == 32 ? p.nwarps : 2 * p.nwarps));
    const int blocks = (groups + threads / 32 - 1) / (threads / 32);
    if (blocks < grid) grid = blocks;
    if constexpr (W >= 32 && !REF) {
        if (p.force_list) {
            const int split = force_split(groups, p.sms);
            if (split > 1) {
                const int cap = p.stack_cap > kSplitQueue ? p.stack_cap : kSplitQueue;
                const size_t sm = force_list_smem_bytes(32 * split, cap);
                if (feat) force_split_kernel<W, PB, true><<<groups, 32 * split, sm, s>>>(p);
                else force_split_kernel<W, PB, false><<<groups, 32 * split, sm, s>>>(p);
                return;
            }
            const size_t sm = force_list_smem_bytes(threads, p.stack_cap);
            if (feat) force_entry<W, false, PB, true, true>()<<<grid, threads, sm, s>>>(p);
            else force_entry<W, false, PB, false, true>()<<<grid, threads, sm, s>>>(p);
            return;
        }
    }
    const size_t sm = force_smem_bytes<W>(threads, p.stack_cap, feat);
    if (feat) force_entry<W, REF, PB, true>()<<<grid, threads, sm, s>>>(p);
    else force_entry<W, REF, PB, false>()<<<grid, threads, sm, s>>>(p);
}

template <int W, bool REF>
static void launch_force_t(const StepParams& p, bool pb, bool feat, int grid, int threads, cudaStream_t s) {
    if (pb) launch_force_pf<W, REF, true>(p, feat, grid, threads, s);
    else launch_force_pf<W, REF, false>(p, feat, grid, threads, s);
}

// Every variant may be launched with up to the largest geometry's shared memory.
template <int W, bool REF, bool PB, bool FEAT>
static cudaError_t prep_force() {
    return cudaFuncSetAttribute(force_entry<W, REF, PB, FEAT>(), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)force_smem_bytes<W>(kForceThreadsMax, kStackCapMax, true));
}

template <int W, bool REF>
static cudaError_t prep_force_w() {
    cudaError_t e = cudaSuccess, t;
    if ((t = prep_force<W, REF, false, false>()) != cudaSuccess) e = t;
    if ((t = prep_force<W, REF, false, true>()) != cudaSuccess) e = t;
    if ((t = prep_force<W, REF, true, false>()) != cudaSuccess) e = t;
    if ((t = prep_force<W, REF, true, true>()) != cudaSuccess) e = t;
    return e;
}

template <int W>
static cudaError_t prep_list_w() {
    cudaError_t e = cudaSuccess, t;
    const int sm = (int)force_list_smem_bytes(kForceThreadsMax, kStackCapMax);
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if ((t = cudaFuncSetAttribute(force_split_kernel<W, false, false>, attr, sm)) != cudaSuccess) e = t;
    if ((t = cudaFuncSetAttribute(force_split_kernel<W, false, true>, attr, sm)) != cudaSuccess) e = t;
    if ((t = cudaFuncSetAttribute(force_split_kernel<W, true, false>, attr, sm)) != cudaSuccess) e = t;
    if ((t = cudaFuncSetAttribute(force_split_kernel<W, true, true>, attr, sm)) != cudaSuccess) e = t;
    if ((t = cudaFuncSetAttribute(force_entry<W, false, false, false, true>(),
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, sm)) != cudaSuccess)
        e = t;
    if ((t = cudaFuncSetAttribute(force_entry<W, false, false, true, true>(),
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, sm)) != cudaSuccess)
        e = t;
    if ((t = cudaFuncSetAttribute(force_entry<W, false, true, false, true>(),
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, sm)) != cudaSuccess)
        e = t;
    if ((t = cudaFuncSetAttribute(force_entry<W, false, true, true, true>(),
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, sm)) != cudaSuccess)
        e = t;
    return e;
}

int prepare_force_kernels() {
    cudaError_t e = cudaSuccess, t;
    if ((t = prep_list_w<32>()) != cudaSuccess) e = t;
    if ((t = prep_list_w<64>()) != cudaSuccess) e = t;
    if ((t = prep_list_w<128>()) != cudaSuccess) e = t;
    if ((t = prep_force_w<128, false>()) != cudaSuccess) e = t;
    if ((t = prep_force_w<64, false>()) != cudaSuccess) e = t;
    if ((t = prep_force_w<32, false>()) != cudaSuccess) e = t;
    if ((t = prep_force_w<32, true>()) != cudaSuccess) e = t;
    if ((t = prep_force_w<16, false>()) != cudaSuccess) e = t;
    if ((t = prep_force_w<16, true>()) != cudaSuccess) e = t;
    return (int)e;
}

bool force_geometry_valid(int vote, int threads, int cap) {
    (void)vote;
    return (threads == 64 || threads == 128 || threads == 256) && cap >= kStackCapMin &&
           cap <= kStackCapMax && cap % 8 == 0;
}

void launch_force(const StepParams& p, int vote, bool ref, bool feat, int grid, int threads, cudaStream_t s) {
    const bool pb = p.theta_body != nullptr;
    if (vote == 128) {
        launch_force_t<128, false>(p, pb, feat, grid, threads, s);  // FMA arithmetic only
    } else if (vote == 64) {
        launch_force_t<64, false>(p, pb, feat, grid, threads, s);   // FMA arithmetic only
    } else if (vote == 16) {
        if (ref) launch_force_t<16, true>(p, pb, feat, grid, threads, s);
        else launch_force_t<16, false>(p, pb, feat, grid, threads, s);
    } else {
        if (ref) launch_force_t<32, true>(p, pb, feat, grid, threads, s);
        else launch_force_t<32, false>(p, pb, feat, grid, threads, s);
    }
}

__global__ void item_order_reset_kernel(int nitems, int* order, int* cost) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nitems; i += gridDim.x * blockDim.x) {
        order[i] = i;
        cost[i] = 0;
    }
}

void launch_item_order_reset(int nitems, int* order, int* cost, cudaStream_t s) {
    if (nitems > 0) item_order_reset_kernel<<<(nitems + 255) / 256, 256, 0, s>>>(nitems, order, cost);
}

int occupancy_force(int vote, bool ref, int threads, int cap, bool list, int* blocks_per_sm) {
    if (list && !ref && vote >= 32) {
        const size_t sm = force_list_smem_bytes(threads, cap);
        if (vote == 128)
            return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, force_entry<128, false, false, false, true>(),
                                                                 threads, sm);
        if (vote == 64)
            return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, force_entry<64, false, false, false, true>(),
                                                                 threads, sm);
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, force_entry<32, false, false, false, true>(),
                                                             threads, sm);
    }
    if (vote == 128)
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, force_kernel<128, false, false, false>,
                                                             threads, force_smem_bytes<128>(threads, cap, false));
    if (vote == 64)
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, force_entry<64, false, false, false>(),
                                                             threads, force_smem_bytes<64>(threads, cap, false));
    if (vote == 16)
        return ref ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, force_kernel<16, true, false, false>,
                                                                   threads, force_smem_bytes<16>(threads, cap, false))
                   : cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, force_kernel<16, false, false, false>,
                                                                   threads, force_smem_bytes<16>(threads, cap, false));
    return ref ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, force_kernel<32, true, false, false>,
                                                               threads, force_smem_bytes<32>(threads, cap, false))
               : cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, force_kernel<32, false, false, false>,
                                                               threads, force_smem_bytes<32>(threads, cap, false));
}

}  // namespace nbh
