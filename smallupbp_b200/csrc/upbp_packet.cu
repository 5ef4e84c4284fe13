// BB1D for packets of camera rays: the queries of path length 1 from one pinhole, 8 x 4 pixels at a time.
//
// A warp that evaluates one query alone walks the tree alone and tests 32 beam pieces at a time, every
// lane with its own piece: the walk, the piece loads and the predicate were three quarters of the BB1D
// time at 1024 x 1024.  The rays of an 8 x 4 pixel block cross nearly the same pieces, so here a block of
// 8 warps takes them together.  It walks the beam-piece LBVH once for their frustum, drops the pieces
// that no ray can take (by the distance of the lines and by which piece holds their closest point), and
// then works in rounds of 1024 pieces: every warp tests 32 pieces against all rays (lane = piece, the
// rays from shared memory, 24 instructions per ray for 32 pairs), which leaves a bit per pair; then the
// warps take the rays in turn and evaluate each ray's pieces 32 at a time, every lane busy and the ray's
// sums in registers.  (A lane per ray instead had 31 of 100 lanes busy, as the rays' work differs, and
// dealing the pairs evenly paid as much for moving between rays.)
//
// What bounds it: instructions, issued in 0.67 of the cycles (ncu, cube512: 7.3 G for 226 M accepted pairs); 24
// warps per SM at 80 registers, and every register that its inner loops spill costs: the L1 that three
// blocks leave is small.  BB1D with the per-query gather beside it (mixed mode), against that gather alone: cube1024
// 269.2 -> 185.4 ms, boxes3 426.6 -> 305.3 ms, cube512 21.2 -> 16.3 ms, the same with KNN radii 12.3 -> 9.8 ms;
// plain mode at cube512 33.5 -> 27.9 ms, at cube1024 542.9 -> 420.4 ms.
//
// The candidate set is the one of the per-query kernels: every accepted pair passes the reference's FP32
// predicate (PhotonBeam.hxx:238-296), the radius test and the reach rule (upbp_device.cuh); the checks
// before them are conservative.  The values are theirs too, but for the rounding of the squared distance
// (bb1d_pair_fast) and of the sums.
#include <algorithm>
#include <cfloat>
#include <cstdint>

#include "upbp_contrib.cuh"
#include "upbp_packet.cuh"

namespace upbp {

namespace {

constexpr float kNan = __builtin_nanf("");
constexpr float kPacketShare = 0.6f;        // k_packet_items
constexpr int kPWarps = 8;                  // warps per block
constexpr int kPThreads = kPWarps * 32;
// The frustum walk pops up to kPNodes nodes a step, two threads per node (one per child).  Its stack
// grows by at most the nodes popped and holds about a step's nodes per tree level; 2048 entries are
// enough that it pops fewer only in the widest frusta (above, one node per step, see below).
constexpr int kPNodes = kPThreads / 2;
constexpr int kPStack = 2048;
constexpr int kPLeaves = 512 + kPThreads;   // leaves waiting: one step finds up to one per thread
constexpr int kPFilter = 4;                 // pieces per thread in one filter pass
constexpr int kPRound = 1024;               // pieces that the rays are evaluated against at a time
constexpr int kPSurv = kPRound + kPFilter * kPThreads;  // pieces waiting for the rays

__device__ __forceinline__ float warp_min(float v)
{
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(kFull, v, o));
    return v;
}
__device__ __forceinline__ float warp_max(float v)
{
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, o));
    return v;
}

// The frustum of a packet's rays: their common origin, the axis k that they advance along (in
// direction sgn), and the ranges of the slopes d_a / |d_k|, d_b / |d_k| along the other two axes.
struct Frustum {
    V3 o;
    int k;
    float sgn, a_lo, a_hi, b_lo, b_hi, k_lo, k_hi;
};

// Component `k`, `k + 1`, `k + 2` (mod 3) of a vector; k is the same for the whole packet.
__device__ __forceinline__ float axis_k(int k, float x, float y, float z) { return k == 0 ? x : (k == 1 ? y : z); }
__device__ __forceinline__ float axis_a(int k, float x, float y, float z) { return k == 0 ? y : (k == 1 ? z : x); }
__device__ __forceinline__ float axis_b(int k, float x, float y, float z) { return k == 0 ? z : (k == 1 ? x : y); }

// The main axis of a direction: k << 1, and 1 for the negative sense.
__device__ __forceinline__ int main_axis(V3 d)
{
    const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    const int k = ax >= ay && ax >= az ? 0 : (ay >= az ? 1 : 2);
    return k << 1 | (axis_k(k, d.x, d.y, d.z) < 0.f ? 1 : 0);
}

// Frustum along `axis` (main_axis) of the rays of the lanes with `valid`, which share the origin o0; false unless
// they have it exactly, have unit directions (the conservative checks assume them) and advance along the axis.
// Warp-wide.  The packet's first ray gives the axis to all of its runs of rays: what holds for the packet then
// holds for each run, whose own first ray may have another main axis.
__device__ __forceinline__ bool packet_frustum(bool valid, V3 o, V3 d, V3 o0, int axis, Frustum& F)
{
    F.o = o0;
    F.k = axis >> 1;
    F.sgn = axis & 1 ? -1.f : 1.f;
    const float dk = axis_k(F.k, d.x, d.y, d.z) * F.sgn;
    const float len2 = d.x * d.x + d.y * d.y + d.z * d.z;
    const bool ok = o.x == o0.x && o.y == o0.y && o.z == o0.z && dk >= 0.4f && fabsf(len2 - 1.f) <= 2e-6f;
    if (__any_sync(kFull, valid && !ok)) return false;
    const float sa = axis_a(F.k, d.x, d.y, d.z) / dk, sb = axis_b(F.k, d.x, d.y, d.z) / dk;
    // widened by the rounding of the slopes
    F.a_lo = warp_min(valid ? sa : FLT_MAX) - 2e-6f;
    F.a_hi = warp_max(valid ? sa : -FLT_MAX) + 2e-6f;
    F.b_lo = warp_min(valid ? sb : FLT_MAX) - 2e-6f;
    F.b_hi = warp_max(valid ? sb : -FLT_MAX) + 2e-6f;
    F.k_lo = warp_min(valid ? dk : FLT_MAX);
    F.k_hi = warp_max(valid ? dk : -FLT_MAX);
    return true;
}

// A work item: the first ray of the run in the order, how many, and the axis of the packet.
__device__ __forceinline__ unsigned long long packet_item(int first, int count, int axis)
{
    return (unsigned long long)(unsigned)first | (unsigned long long)(count | axis << 8) << 32;
}

// Whether the frustum between the depths z0 >= 0 and z1 along its axis can meet the box.
__device__ __forceinline__ bool frustum_box(const Frustum& F, float z0, float z1, float lx, float ly, float lz,
                                            float hx, float hy, float hz)
{
    const float ok = axis_k(F.k, F.o.x, F.o.y, F.o.z);
    const float u = (axis_k(F.k, lx, ly, lz) - ok) * F.sgn, v = (axis_k(F.k, hx, hy, hz) - ok) * F.sgn;
    const float zl = fmaxf(fminf(u, v), z0), zh = fminf(fmaxf(u, v), z1);
    const float oa = axis_a(F.k, F.o.x, F.o.y, F.o.z), ob = axis_b(F.k, F.o.x, F.o.y, F.o.z);
    const float amin = fminf(zl * F.a_lo, zh * F.a_lo), amax = fmaxf(zl * F.a_hi, zh * F.a_hi);
    const float bmin = fminf(zl * F.b_lo, zh * F.b_lo), bmax = fmaxf(zl * F.b_hi, zh * F.b_hi);
    return !(zl > zh) && !(amin > axis_a(F.k, hx, hy, hz) - oa) && !(amax < axis_a(F.k, lx, ly, lz) - oa) &&
           !(bmin > axis_b(F.k, hx, hy, hz) - ob) && !(bmax < axis_b(F.k, lx, ly, lz) - ob);
}

// The sum over the axes of the largest distance from the origin to the beams' box (a bound of
// |O2 - O1|), and the largest coordinate in play: the scales of the conservative margins.
__device__ __forceinline__ void packet_scales(V3 o, const float* __restrict__ bb, float& reach, float& coord)
{
    reach = fmaxf(fabsf(bb[0] - o.x), fabsf(bb[3] - o.x)) + fmaxf(fabsf(bb[1] - o.y), fabsf(bb[4] - o.y)) +
            fmaxf(fabsf(bb[2] - o.z), fabsf(bb[5] - o.z));
    coord = fmaxf(fmaxf(fabsf(o.x), fabsf(o.y)), fmaxf(fabsf(o.z), 1.f));
    for (int c = 0; c < 6; ++c) coord = fmaxf(coord, fabsf(bb[c]));
}

// ----------------------------------------------------------------- packets of an image
// The pixel blocks (8 x 4) of the queries: a block's camera rays are consecutive in the pixel order, whose keys'
// low five bits count the pixels of an aligned block (the other segments' keys have bit 29).  A warp takes the
// blocks that begin at its 32 places of the order, one after the other, so the work grows with the
// queries, not with the image.  A block's rays form a packet if there are at most 32 of them, they make a
// frustum, and that is at most max_width across at its far end: the rays of a frustum much wider than the beam
// pieces share few of them.  The packets are listed in no particular order.
__global__ void __launch_bounds__(256) k_packet_setup(const SegQueriesDev Q, const uint32_t* __restrict__ keys,
                                                      const int32_t* __restrict__ order,
                                                      const uint32_t* __restrict__ cnt_pb2d,
                                                      int64_t n_pixels, const float* __restrict__ bbox, float max_width,
                                                      int2* range, uint32_t* weight, uint8_t* in_packet,
                                                      PacketTotals* totals)
{
    constexpr uint32_t kNoBlock = 0xffffffffu;
    const int n = (int)Q.n;
    const int base = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) & ~31ll), lane = threadIdx.x & 31;
    if (base >= n) return;
    const auto block_of = [&](int i) {
        const uint32_t k = i < n ? __ldg(&keys[i]) : kNoBlock;
        return k < (1u << 28) ? k >> 5 : kNoBlock;
    };
    const int i = base + lane;
    const uint32_t mine = block_of(i), before = i > 0 ? block_of(i - 1) : kNoBlock;
    if (mine != kNoBlock && block_of(i + 1) == kNoBlock) totals->camera = (unsigned)i + 1u;
    unsigned starts = __ballot_sync(kFull, mine != kNoBlock && mine != before);
    for (; starts; starts &= starts - 1) {
        const int from = __ffs(starts) - 1, start = base + from;
        const uint32_t block = __shfl_sync(kFull, mine, from);
        const unsigned members = __ballot_sync(kFull, block_of(start + lane) == block);
        const int count = __popc(members);
        bool ok = !(count == 32 && block_of(start + 32) == block);
        const bool valid = lane < count;
        const int64_t q = valid ? (int64_t)__ldg(&order[start + lane]) : 0;
        V3 o = v3(0.f, 0.f, 0.f), d = o;
        float lo = FLT_MAX, hi = 0.f;
        unsigned w = 0;
        if (valid && ok) {
            o = v3(Q.origin[3 * q], Q.origin[3 * q + 1], Q.origin[3 * q + 2]);
            d = v3(Q.direction[3 * q], Q.direction[3 * q + 1], Q.direction[3 * q + 2]);
            const int sb = Q.seg_begin[q], sc = Q.seg_count[q];
            for (int k = 0; k < sc; ++k) {
                lo = fminf(lo, Q.seg_dist_min[sb + k]);
                hi = fmaxf(hi, Q.seg_dist_max[sb + k]);
            }
            w = cnt_pb2d ? min(__ldg(&cnt_pb2d[q]), 1u << 24) : 0u;
        }
        Frustum F;
        const V3 o0 = v3(__shfl_sync(kFull, o.x, 0), __shfl_sync(kFull, o.y, 0), __shfl_sync(kFull, o.z, 0));
        const int axis = __shfl_sync(kFull, main_axis(d), 0);
        ok = packet_frustum(valid, o, d, o0, axis, F) && ok;
        ok = __all_sync(kFull, !valid || (lo >= 0.f && Q.pixel[q] < n_pixels)) && ok;
        if (ok) {
            float reach, coord;
            packet_scales(F.o, bbox, reach, coord);
            ok = fmaxf(F.a_hi - F.a_lo, F.b_hi - F.b_lo) * fminf(warp_max(hi), reach) <= max_width;
        }
        w = __reduce_add_sync(kFull, w);
        if (!ok) continue;
        if (valid) in_packet[q] = 1;
        if (lane == 0) {
            const unsigned p = atomicAdd(&totals->packets, 1u);
            range[p] = make_int2(start, count | axis << 8);
            weight[p] = w + 1u;  // the work estimate (PB2D candidates)
            atomicAdd(&totals->rays, (unsigned)count);
            atomicAdd(&totals->weight, (unsigned long long)w + 1ull);
        }
    }
}

// The work items: a packet, or 2 to 8 equal runs of its rays where the whole would be more than `share` of
// all work (the heaviest packet has 15 times the mean's work, and in a small image a packet's block
// would run long after the others are done).  Each item is a packet of its own, with a narrower frustum,
// but walks the tree again: at cube512 a share of 0.05 / 0.25 / 0.6 / 1 of what a resident block gets
// on average took 18.4 / 15.7 / 14.9 / 15.0 ms (an earlier version).  The items are sorted by weight; slots
// without one have 0 (the caller's).  A packet of P parts has more than share P / 2 of the weight, so that there
// are at most 2 / share items more than packets.
__global__ void __launch_bounds__(256) k_packet_items(const uint32_t* __restrict__ weight, const int2* __restrict__ range,
                                                      float share, unsigned slots, PacketTotals* totals, uint32_t* key,
                                                      unsigned long long* item)
{
    const unsigned p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= totals->packets || totals->camera < kPacketCamera) return;
    if (p == 0) totals->queries = totals->rays;
    const uint32_t w = weight[p];
    const int2 r = range[p];
    const int count = r.y & 0xff;
    const float limit = share * (float)totals->weight;
    int log = 0;
    while (1 << log < kPacketParts && (float)w > limit * (float)(1 << log) && 2 << log <= count) ++log;
    const unsigned at = atomicAdd(&totals->items, 1u << log);
    for (int k = 0; k < 1 << log; ++k) {
        const int from = (count * k) >> log, to = (count * (k + 1)) >> log;
        if (at + k >= slots) return;  // cannot happen (see above); kept as a guard
        key[at + k] = max(1u, w >> log);
        item[at + k] = packet_item(r.x + from, to - from, r.y >> 8);
    }
}


// ----------------------------------------------------------------- the gather
// What the walk needs of the packet.
struct PacketWalk {
    Frustum F;
    float ac, ah, bc, bh;     // middle and half width of the slopes
    float dir2_lo, dir2_hi;   // |(slope a, slope b, 1)|^2 over the frustum
    float z0, z1;             // depths of the segment
    // margins of the tests in approximate arithmetic: the squared distance of the lines (a few ulp of
    // |O2 - O1|), and the beam parameter of their closest points times 1 - (d.d2)^2.  The latter is a few ulp of
    // |O2 - O1| too, and 6e-6 of the coordinates: the predicate takes a pair by its own t1, which is off by up to
    // that (piece_takes_fast), so the lines' closest point may lie that far beyond the ray's end, where the
    // owner is the piece opposite the end.
    float near_eps, u_eps;
    float reach;              // bound of |O2 - O1|_1
    float coord, scale;       // largest coordinate; that and the end of the segment
    float piece_len;          // longest piece
    unsigned active;          // the rays with this segment in a scattering medium
    bool one_medium;          // all of them in medium mid0: the other media's pieces are dropped
    int mid0;
    int sp, nleaf, nsurv, lpos;  // the walk's lists
    int n_rays;
};

struct PacketShared {
    PacketWalk walk;
    DMedium media[UPBP_MAX_MEDIA];
    // per ray, written by warp 0: the query (-1: no ray), its first segment, how many and which one is in
    // hand, and what the segments before pass on (segment_loop)
    int64_t ray_q[32];
    int ray_sb[32], ray_sc[32], ray_at[32];
    float attn_r[32], attn_g[32], attn_b[32], rsp[32], rsr[32];
    float4 ray_d[32];            // direction, dmin
    float4 ray_s[32];            // dmax, mRaySamplePdf, mRaySampleRevPdf, last_pdf_w_inv
    int ray_i[32];               // medium | raySamplingFlags << 8
    // per ray: the result, in the segment (the rounds' sums, in FP64: a running FP32 sum of them would round more
    // than the 32 sums of a warp's lanes do) and of all segments
    double acc_r[32], acc_g[32], acc_b[32];
    float sum_r[32], sum_g[32], sum_b[32];
    unsigned cnt[32];
    unsigned long long hash[32];
    // the pieces in hand: which, their candidate hash, and per 32 of them and ray those the ray can meet
    int surv[kPSurv];
    unsigned long long surv_hash[kPRound];
    unsigned mask[kPRound / 32][32];
    int slow[32][64];            // per ray: pieces whose pair FP32 does not decide
    int slow_n[32];
    uint16_t list[kPWarps][kPRound];  // per warp: the pieces of the ray that it evaluates
    int stack[kPStack];
    int leaves[kPLeaves];
    int count[kPWarps];
    unsigned next, next_ray;
};

// Lane = piece: which of the pieces [first, first + 32) of the list each ray can meet.  One warp.
__device__ __forceinline__ void packet_test(const GatherConsts& K, const BeamBVH& B, PacketShared& S, int first, int n)
{
    const int lane = threadIdx.x & 31;
    const PacketWalk& P = S.walk;
    const float near_eps = P.near_eps, u_eps = P.u_eps;
    const float half_len = 0.5f * P.piece_len * 1.00001f + 0.03f * u_eps;
    // a: n = d2 x (O2 - O1), 1.002 max radius^2;  b: direction, slack and margin;  c: p = (O2 - O1) - ew d2,
    // ew + middle of the piece
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a, c = a;
    bool use = false;
    float near = 0.f;
    if (lane < n) {
        const int p = S.surv[first + lane];
        const float4 pa = __ldg(&B.pa[p]), pb = __ldg(&B.pb[p]), pc = __ldg(&B.pc[p]);
        const V3 w = v3(pa.x - P.F.o.x, pa.y - P.F.o.y, pa.z - P.F.o.z);
        const float ew = pb.x * w.x + pb.y * w.y + pb.z * w.z;
        const float len2 = pb.x * pb.x + pb.y * pb.y + pb.z * pb.z;
        use = !(P.one_medium && __float_as_int(pc.w) != P.mid0);
        // a direction that is no unit vector passes the test (and its piece is marked, as ~piece): the exact
        // predicate decides
        const bool unit = fabsf(len2 - 1.f) <= 2e-6f;
        if (unit) a = make_float4(pb.y * w.z - pb.z * w.y, pb.z * w.x - pb.x * w.z, pb.x * w.y - pb.y * w.x, 1.002f * pb.w);
        else S.surv[first + lane] = ~p;
        near = fmaf(a.w, 2e-5f, near_eps);
        b = make_float4(pb.x, pb.y, pb.z, unit ? u_eps + piece_slack(pa.w, pb.w, pc.x, pc.y, K.bb1d_extra) : FLT_MAX);
        c = make_float4(w.x - ew * pb.x, w.y - ew * pb.y, w.z - ew * pb.z,
                        pc.y - pc.x <= P.piece_len * 1.00001f ? ew + 0.5f * (pc.x + pc.y) : kNan);
        S.surv_hash[first + lane] = mix64((unsigned long long)__float_as_int(pc.z));
    }
    unsigned word = 0;
    const int rays = P.n_rays;
#pragma unroll 4
    for (int r = 0; r < rays; ++r) {
        const float4 d = S.ray_d[r];
        const float ad = d.x * a.x + d.y * a.y + d.z * a.z;
        const float cs = d.x * b.x + d.y * b.y + d.z * b.z;
        const float pd = d.x * c.x + d.y * c.y + d.z * c.z;
        const float om = fmaf(-cs, cs, 1.f);
        // the lines' distance (the predicate's first check), then the beam parameter of their closest
        // points inside the piece, |u - middle| <= half + margin / om + slack / sqrt(om), times om
        const bool hit = use && !(ad * ad > fmaf(a.w, om, near)) &&
                         !(fabsf(fmaf(cs, pd, -c.w * om)) > fmaf(half_len, om, b.w));
        const unsigned vote = __ballot_sync(kFull, hit);
        if (lane == r) word = vote;
    }
    S.mask[first >> 5][lane] = word;
}

// A load that stays where it is written: what only the contribution needs is read there, or it would take the
// pair's registers (cube1024 193.2 -> 187.9 ms).
__device__ __forceinline__ float4 ld_shared(const float4* p)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"((unsigned)__cvta_generic_to_shared(p)));
    return v;
}

// One ray, lane = piece: evaluates the pieces that it can meet, 32 at a time.  Pairs that FP32 does not
// decide (2 % of them) wait in the ray's list until there are 32, or until the segment ends (flush): the
// exact predicate, the FP64 closest points and their divergence are paid for once in 32 pairs.
template <bool kMixed>
__device__ __forceinline__ void packet_ray(const GatherConsts& K, const LightSoA& Lv, const BeamBVH& B, const BeamSoA& Bs,
                                           PacketShared& S, int r, int groups, uint16_t* list, bool flush)
{
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    // ---- the pieces, in the order of the list
    const unsigned bits0 = lane < groups ? S.mask[lane][r] : 0u;
    int at = __popc(bits0);
    const int own = at;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(kFull, at, d);
        if (lane >= d) at += v;
    }
    const int total = __shfl_sync(kFull, at, 31);
    int sn = S.slow_n[r];
    if (total == 0 && !(flush && sn > 0)) return;
    at -= own;
    for (unsigned bits = bits0; bits; bits &= bits - 1) list[at++] = (uint16_t)(lane * 32 + __ffs(bits) - 1);
    __syncwarp();
    // ---- the ray (the same in every lane); a camera path of length 1 has no earlier vertices
    const upbp_mis no_mis{};
    const CamSum no_sum{};
    SegCtx s;
    {
        const float4 rd = S.ray_d[r], rs = S.ray_s[r];
        s.o = S.walk.F.o;
        s.d = v3(rd.x, rd.y, rd.z);
        s.dmin = rd.w;
        s.dmax = rs.x;
        s.rsf = (uint32_t)S.ray_i[r] >> 8;
        s.L = 1;
        s.ray_flags = K.P.query_beam_type | K.P.techniques;
        s.cam = nullptr;
        s.e = &no_mis;
        s.cs = &no_sum;
    }
    const int mid = S.ray_i[r] & 0xff;
    const DMedium& m = S.media[mid];
    Rgb part = rgb(0.f);
    unsigned cnt = 0;
    unsigned long long h = 0;
    int base = 0;
    for (;;) {
        // the slow list first when it is full (or at the end); its order in the sum is fixed as well
        const bool slow = sn >= 32 || (base >= total && flush && sn > 0);
        if (!slow && base >= total) break;
        int piece = -1;
        bool unit = true;
        unsigned long long hp = 0;
        if (slow) {
            const int n = min(sn, 32);
            sn -= n;
            if (lane < n) piece = S.slow[r][sn + lane];
        } else {
            const int k = base + lane;
            base += 32;
            if (k < total) {
                const int i = list[k];
                piece = S.surv[i];
                hp = S.surv_hash[i];
                unit = piece >= 0;
                piece = unit ? piece : ~piece;
            }
        }
        bool undecided = false;
        if (piece >= 0) {
            const float4 pa = __ldg(&B.pa[piece]), pb = __ldg(&B.pb[piece]), pc = __ldg(&B.pc[piece]);
            const V3 o2 = v3(pa.x, pa.y, pa.z), d2 = v3(pb.x, pb.y, pb.z);
            const int beam = __float_as_int(pc.z);
            PiecePayload py;
            if (kMixed) py.lv = __ldg(&B.pay[piece].lv);
            const float rs = Bs.rchange ? (kMixed ? py.lv.z : __ldg(&Bs.radius[beam])) : Bs.radius_const;
            const float rc = Bs.rchange ? __ldg(&Bs.rchange[beam]) : 0.f;
            PairGeo pg;
            float dist = 0.f, sinT = 0.f;
            int take = 0;
            if (kMixed) {
                if (slow) {
                    take = pair_slow(s.o, s.d, s.dmin, s.dmax, o2, d2, pa.w, pb.w, pc.x, pc.y, rs, rc, K.bb1d_extra, pg);
                    hp = mix64((unsigned long long)beam);
                } else {
                    // d1.O1 and the scale are taken anew, for the registers (cube1024 187.9 -> 184.8 ms)
                    take = bb1d_pair_fast(s.o, s.d, xdot3(s.d, s.o), s.dmin, s.dmax, o2, d2, pa.w, pb.w, pc.x, pc.y,
                                          S.walk.reach, fmaxf(S.walk.scale, pa.w), rs, rc, pg);
                    if (!unit) take = -1;
                }
            } else {
                float e;
                if (test_beam_beam(s.o, s.d, s.dmin, s.dmax, o2, d2, 0.f, pa.w, pb.w, &dist, &sinT, &pg.t1, &pg.u, &pg.cosb,
                                   &e) &&
                    !(radius_at(rs, rc, pg.u) < dist))  // PhotonBeam.hxx:411-413
                    take = piece_takes_fast(s.o, s.d, s.dmin, s.dmax, o2, pa.w, pc.x, pc.y, pg.t1, pg.cosb, e, dist, rs,
                                            rc, K.bb1d_extra);
                if (slow) {
                    if (take < 0)
                        take = piece_takes_f64(s.o, s.d, s.dmin, s.dmax, o2, d2, pa.w, pc.x, pc.y, rs, rc, K.bb1d_extra);
                    hp = mix64((unsigned long long)beam);
                }
            }
            undecided = take < 0;
            if (take > 0 && __float_as_int(pc.w) == mid) {  // mMedium == medium (PhotonBeam.hxx:390)
                ++cnt;
                h += hp;
                const float radius = radius_at(rs, rc, pg.u);
                const float4 rs4 = ld_shared(&S.ray_s[r]);  // dmax, mRaySamplePdf, mRaySampleRevPdf, last_pdf_w_inv
                s.rs_pdf = rs4.y;
                s.rs_rev_pdf = rs4.z;
                s.last_pdf_w_inv = rs4.w;
                if (kMixed) {  // loaded here for the registers as well
                    py.thr = __ldg(&B.pay[piece].thr);
                    py.pdf = __ldg(&B.pay[piece].pdf);
                    part = part + bb1d_contrib_packed<true>(K, m, s, py, pg, radius);
                } else {
                    part = part + bb1d_contrib<false>(K, m, Lv, Bs, s, beam, o2, d2, radius, dist, sinT, pg.t1, pg.u);
                }
            }
        }
        const unsigned vote = __ballot_sync(kFull, undecided);
        if (vote) {
            if (undecided) S.slow[r][sn + __popc(vote & lt)] = piece;
            sn += __popc(vote);
            __syncwarp();
        }
    }
    const float x = warp_sum(part.r), y = warp_sum(part.g), z = warp_sum(part.b);
    cnt = __reduce_add_sync(kFull, cnt);
    h = warp_sum_u64(h);
    if (lane == 0) {
        S.acc_r[r] += x;
        S.acc_g[r] += y;
        S.acc_b[r] += z;
        S.cnt[r] += cnt;
        S.hash[r] += h;
        S.slow_n[r] = sn;
    }
    __syncwarp();
}

// The walk: fills the list of pieces near the frustum from the LBVH, as far as there is room.  Block-wide.
__device__ __forceinline__ void packet_walk(const GatherConsts& K, const BeamBVH& B, PacketShared& S)
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int leaf_shift = __ffs(B.leaf) - 1;
    const PacketWalk& P = S.walk;
    int sp = P.sp, nleaf = P.nleaf, nsurv = P.nsurv, lpos = P.lpos;
    __syncthreads();
    while (nsurv < kPRound) {
        if (lpos < (nleaf << leaf_shift)) {
            // one filter pass: the pieces whose line comes within their radius of the frustum
            const Frustum& F = P.F;
            unsigned keep = 0, votes[kPFilter];
            int ids[kPFilter], mine = 0;
#pragma unroll
            for (int f = 0; f < kPFilter; ++f) {
                const int idx = lpos + (warp * kPFilter + f) * 32 + lane;
                int p = -1;
                if (idx < (nleaf << leaf_shift)) {
                    p = (S.leaves[idx >> leaf_shift] << leaf_shift) + (idx & ((1 << leaf_shift) - 1));
                    if (p >= B.n) p = -1;
                }
                ids[f] = p;
                bool hit = false;
                if (p >= 0) {
                    const float4 pa = __ldg(&B.pa[p]), pb = __ldg(&B.pb[p]);
                    const V3 w = v3(pa.x - F.o.x, pa.y - F.o.y, pa.z - F.o.z);
                    const float nx = pb.y * w.z - pb.z * w.y, ny = pb.z * w.x - pb.x * w.z,
                                nz = pb.x * w.y - pb.y * w.x;
                    const float na = axis_a(F.k, nx, ny, nz), nb = axis_b(F.k, nx, ny, nz);
                    const float da = axis_a(F.k, pb.x, pb.y, pb.z), db = axis_b(F.k, pb.x, pb.y, pb.z);
                    const float mn = na * P.ac + nb * P.bc + axis_k(F.k, nx, ny, nz) * F.sgn;
                    const float md = da * P.ac + db * P.bc + axis_k(F.k, pb.x, pb.y, pb.z) * F.sgn;
                    const float least = fmaxf(0.f, fabsf(mn) - (fabsf(na) * P.ah + fabsf(nb) * P.bh));
                    const float dmn = fmaxf(0.f, fabsf(md) - (fabsf(da) * P.ah + fabsf(db) * P.bh));
                    const float len2 = pb.x * pb.x + pb.y * pb.y + pb.z * pb.z;
                    const float s2 = fmaf(-dmn, dmn, P.dir2_hi) + 1e-4f;
                    const bool unit = fabsf(len2 - 1.f) <= 2e-6f;
                    hit = !(least * least > fmaf(1.002f * pb.w, s2, 8.f * P.near_eps)) || !unit;
                    // the beam parameter u = (d.d2)(d.p) / (d.d - (d.d2)^2) - ew of the closest
                    // points over the frustum's directions d, in interval arithmetic
                    const float br = fabsf(da) * P.ah + fabsf(db) * P.bh;
                    const float om_lo = P.dir2_lo - (fabsf(md) + br) * (fabsf(md) + br);
                    if (hit && unit && om_lo > 0.01f) {
                        const float4 pc = __ldg(&B.pc[p]);
                        const float ew = pb.x * w.x + pb.y * w.y + pb.z * w.z;
                        const float px = w.x - ew * pb.x, py = w.y - ew * pb.y, pz = w.z - ew * pb.z;
                        const float pm_a = axis_a(F.k, px, py, pz), pm_b = axis_b(F.k, px, py, pz);
                        const float pm = pm_a * P.ac + pm_b * P.bc + axis_k(F.k, px, py, pz) * F.sgn;
                        const float pr = fabsf(pm_a) * P.ah + fabsf(pm_b) * P.bh;
                        const float x = md * pm, xr = fabsf(md) * pr + (fabsf(pm) + pr) * br;
                        const float r_lo = 1.f / s2, r_hi = 1.f / om_lo;
                        const float u_lo = (x - xr) * (x < xr ? r_hi : r_lo) - ew;
                        const float u_hi = (x + xr) * (x > -xr ? r_hi : r_lo) - ew;
                        const float room = P.u_eps * P.dir2_hi * r_hi +
                                           piece_slack(pa.w, pb.w, pc.x, pc.y, K.bb1d_extra) * sqrtf(P.dir2_hi * r_hi);
                        hit = !(u_hi < pc.x - room) && !(u_lo > pc.y + room);
                    }
                }
                votes[f] = __ballot_sync(kFull, hit);
                if (hit) keep |= 1u << f;
                mine += __popc(votes[f]);
            }
            if (lane == 0) S.count[warp] = mine;
            __syncthreads();
            int at = nsurv, all = 0;
#pragma unroll
            for (int v = 0; v < kPWarps; ++v) {
                const int n = S.count[v];
                if (v < warp) at += n;
                all += n;
            }
#pragma unroll
            for (int f = 0; f < kPFilter; ++f) {
                if (keep & (1u << f)) S.surv[at + __popc(votes[f] & lt)] = ids[f];
                at += __popc(votes[f]);
            }
            nsurv += all;
            lpos += kPFilter * kPThreads;
            __syncthreads();
            continue;
        }
        nleaf = lpos = 0;
        if (sp == 0) break;
        // the stack stays within its bound as in warp_traverse: a step pops at most what
        // keeps it there, one node (a depth-first walk) above that
        while (sp > 0 && nleaf <= kPLeaves - kPThreads) {
            const int take = min(min(sp, kPNodes), max(1, kPStack - kMaxTreeDepth - sp));
            int child = 0;
            bool hit = false;
            if ((tid >> 1) < take) {
                const BNode* nd = &B.nodes[S.stack[sp - 1 - (tid >> 1)]];
                const bool right = tid & 1;
                const float4 u = __ldg(right ? &nd->b : &nd->a), v = __ldg(right ? &nd->c : &nd->b);
                child = __ldg(right ? &nd->d.y : &nd->d.x);
                hit = right ? frustum_box(P.F, P.z0, P.z1, u.z, u.w, v.x, v.y, v.z, v.w)
                            : frustum_box(P.F, P.z0, P.z1, u.x, u.y, u.z, u.w, v.x, v.y);
            }
            const unsigned push = __ballot_sync(kFull, hit && child >= 0);
            const unsigned leaf = __ballot_sync(kFull, hit && child < 0);
            if (lane == 0) S.count[warp] = __popc(push) | (__popc(leaf) << 16);
            __syncthreads();
            int before = 0, all = 0;
#pragma unroll
            for (int v = 0; v < kPWarps; ++v) {
                const int n = S.count[v];
                if (v < warp) before += n;
                all += n;
            }
            sp -= take;
            if (hit && child >= 0) S.stack[sp + (before & 0xffff) + __popc(push & lt)] = child;
            if (hit && child < 0) S.leaves[nleaf + (before >> 16) + __popc(leaf & lt)] = ~child;
            sp += all & 0xffff;
            nleaf += all >> 16;
            __syncthreads();
        }
    }
    if (tid == 0) {
        S.walk.sp = sp;
        S.walk.nleaf = nleaf;
        S.walk.nsurv = nsurv;
        S.walk.lpos = lpos;
    }
    __syncthreads();
}

// The rays and the frustum (along `axis`) of a run rg of a packet's rays, by warp 0 (lane = ray).
__device__ __forceinline__ void packet_begin(const SegQueriesDev& Q, const int32_t* __restrict__ order, int2 rg, int axis,
                                             const float* __restrict__ bbox, float piece_len, PacketShared& S)
{
    const int lane = threadIdx.x & 31;
    const bool valid = lane < rg.y;
    const int64_t q = valid ? (int64_t)__ldg(&order[rg.x + lane]) : -1;
    V3 o = v3(0.f, 0.f, 0.f), d = o;
    float lpw = 0.f;
    int sb = 0, sc = 0;
    if (valid) {
        o = v3(Q.origin[3 * q], Q.origin[3 * q + 1], Q.origin[3 * q + 2]);
        d = v3(Q.direction[3 * q], Q.direction[3 * q + 1], Q.direction[3 * q + 2]);
        lpw = Q.last_pdf_w_inv[q];
        if (Q.flags[q] & UPBP_Q_BB1D) {
            sb = Q.seg_begin[q];
            sc = Q.seg_count[q];
        }
    }
    PacketWalk P;
    const V3 o0 = v3(__shfl_sync(kFull, o.x, 0), __shfl_sync(kFull, o.y, 0), __shfl_sync(kFull, o.z, 0));
    packet_frustum(valid, o, d, o0, axis, P.F);
    packet_scales(P.F.o, bbox, P.reach, P.coord);
    P.near_eps = 4.7e-9f * P.reach * P.reach;
    P.u_eps = 3.5e-5f * P.reach + 6e-6f * P.coord;
    P.piece_len = piece_len;
    const Frustum& F = P.F;
    P.ac = 0.5f * (F.a_lo + F.a_hi), P.ah = 0.5f * (F.a_hi - F.a_lo) + 1e-7f;
    P.bc = 0.5f * (F.b_lo + F.b_hi), P.bh = 0.5f * (F.b_hi - F.b_lo) + 1e-7f;
    const float a_in = F.a_lo > 0.f ? F.a_lo : (F.a_hi < 0.f ? -F.a_hi : 0.f);
    const float b_in = F.b_lo > 0.f ? F.b_lo : (F.b_hi < 0.f ? -F.b_hi : 0.f);
    P.dir2_lo = (1.f + a_in * a_in + b_in * b_in) * 0.99998f;
    P.dir2_hi = (1.f + fmaxf(F.a_lo * F.a_lo, F.a_hi * F.a_hi) + fmaxf(F.b_lo * F.b_lo, F.b_hi * F.b_hi)) * 1.00002f;
    P.active = 0;
    P.n_rays = rg.y;
    if (lane == 0) S.walk = P;
    S.ray_q[lane] = q;
    S.ray_sb[lane] = sb;
    S.ray_sc[lane] = sc;
    S.ray_at[lane] = 0;
    S.attn_r[lane] = S.attn_g[lane] = S.attn_b[lane] = S.rsp[lane] = S.rsr[lane] = 1.f;
    S.sum_r[lane] = S.sum_g[lane] = S.sum_b[lane] = 0.f;
    S.cnt[lane] = 0;
    S.hash[lane] = 0;
    S.ray_d[lane] = make_float4(d.x, d.y, d.z, 0.f);
    S.ray_s[lane] = make_float4(0.f, 0.f, 0.f, lpw);
}

// What segment i of a ray passes on to its later ones (segment_loop).  Lane = ray.
__device__ __forceinline__ void packet_pass_on(const GatherConsts& K, const SegQueriesDev& Q, int i, PacketShared& S)
{
    const int lane = threadIdx.x & 31;
    const int64_t q = S.ray_q[lane];
    const uint32_t qf = Q.flags[q];
    const int sg = S.ray_sb[lane] + i;
    const DMedium& m = S.media[Q.seg_medium[sg]];
    Rgb attn{S.attn_r[lane], S.attn_g[lane], S.attn_b[lane]};
    float pdf, rev;
    if (qf & UPBP_Q_LITE) {
        const float dmin = Q.seg_dist_min[sg], dmax = Q.seg_dist_max[sg];
        attn = attn * eval_att(m, dmax - dmin);
        pdf = ray_sample_pdf(m, dmin, dmax, i == 0 && (qf & UPBP_Q_ORIGIN_IN_MEDIUM) ? UPBP_ORIGIN_IN_MEDIUM : 0u, &rev);
    } else {
        const Rgb sa{Q.seg_attenuation[3 * sg], Q.seg_attenuation[3 * sg + 1], Q.seg_attenuation[3 * sg + 2]};
        pdf = Q.seg_pdf[sg];
        rev = Q.seg_rev_pdf[sg];
        attn = attn * (K.P.query_beam_type == UPBP_SHORT_BEAM ? sa / pdf : sa);
    }
    S.rsp[lane] *= pdf;
    S.rsr[lane] *= rev;
    S.attn_r[lane] = attn.r;
    S.attn_g[lane] = attn.g;
    S.attn_b[lane] = attn.b;
    if (!rgb_positive(attn)) S.ray_sc[lane] = 0;
}

// The next scattering segment of every ray, by warp 0, and the start of its walk.  Each ray has its own
// place in its list: a ray that scatters in the medium lists fewer segments before it than one that
// passes through, and taken by their index the two would need a walk each.
__device__ __forceinline__ void packet_segment(const GatherConsts& K, const SegQueriesDev& Q, int n_leaves,
                                               PacketShared& S)
{
    const int lane = threadIdx.x & 31;
    const int64_t q = S.ray_q[lane];
    const int sb = S.ray_sb[lane];
    int i = S.ray_at[lane];
    if ((S.walk.active >> lane) & 1u) packet_pass_on(K, Q, i++, S);  // the segment before
    __syncwarp();
    while (i < S.ray_sc[lane] && !S.media[Q.seg_medium[sb + i]].has_scat) packet_pass_on(K, Q, i++, S);
    S.ray_at[lane] = i;
    const bool active = i < S.ray_sc[lane];
    const int mid = active ? Q.seg_medium[sb + i] : 0;
    const float dmin = active ? Q.seg_dist_min[sb + i] : 0.f, dmax = active ? Q.seg_dist_max[sb + i] : 0.f;
    const uint32_t inside = active && i == 0 && (Q.flags[q] & UPBP_Q_ORIGIN_IN_MEDIUM) ? UPBP_ORIGIN_IN_MEDIUM : 0u;
    const unsigned act = __ballot_sync(kFull, active);
    const int mid0 = __shfl_sync(kFull, mid, act ? __ffs(act) - 1 : 0);
    const bool one_medium = __all_sync(kFull, !active || mid == mid0);
    const float near = warp_min(active ? dmin : FLT_MAX), far = warp_max(active ? dmax : 0.f);
    const float4 rd = S.ray_d[lane], rs = S.ray_s[lane];
    S.ray_d[lane] = make_float4(rd.x, rd.y, rd.z, dmin);
    S.ray_s[lane] = make_float4(dmax, S.rsp[lane], S.rsr[lane], rs.w);
    S.ray_i[lane] = mid | (int)((UPBP_END_IN_MEDIUM | inside) << 8);
    if (lane == 0) {
        PacketWalk& P = S.walk;
        P.scale = fmaxf(P.coord, far);
        P.active = act;
        P.one_medium = one_medium;
        P.mid0 = mid0;
        P.z0 = fmaxf(0.f, near * P.F.k_lo - K.eps);
        P.z1 = far * P.F.k_hi + K.eps;
        P.nsurv = P.lpos = 0;
        P.nleaf = n_leaves == 1 ? 1 : 0;
        P.sp = 1 - P.nleaf;
        S.leaves[0] = S.stack[0] = 0;
        S.next_ray = 0;
    }
    S.acc_r[lane] = S.acc_g[lane] = S.acc_b[lane] = 0.0;
    S.slow_n[lane] = 0;
}

// Persistent: a block takes the next item from the work counter.  kMinBlocks blocks of 8 warps per SM.
// What outlives a step is kept in shared memory: the evaluation needs the registers.
template <bool kMixed, int kMinBlocks>
__global__ void __launch_bounds__(kPThreads, kMinBlocks)
k_bb1d_packet(const __grid_constant__ GatherConsts K, const __grid_constant__ LightSoA Lv,
              const __grid_constant__ BeamBVH B, const __grid_constant__ BeamSoA Bs, const SegQueriesDev Q,
              const Outputs O, const int32_t* __restrict__ order, const unsigned long long* __restrict__ items,
              const PacketTotals* __restrict__ totals,
              const float* __restrict__ bbox, float piece_len, unsigned* work)
{
    extern __shared__ __align__(16) unsigned char smem[];
    PacketShared& S = *reinterpret_cast<PacketShared*>(smem);
    asm volatile("griddepcontrol.launch_dependents;");  // the gather per query may start beside this one
    stage_media(K, S.media);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (;;) {
        if (warp == 0) {
            if (lane == 0) S.next = atomicAdd(work, 1u);
            __syncwarp();
            if (S.next < totals->items) {
                const unsigned long long it = items[S.next];
                packet_begin(Q, order, make_int2((int)(unsigned)it, (int)(it >> 32) & 0xff), (int)(it >> 40), bbox, piece_len,
                             S);
            }
        }
        __syncthreads();
        if (S.next >= totals->items) break;
        for (;;) {
            if (warp == 0) packet_segment(K, Q, B.n_leaves, S);
            __syncthreads();
            if (S.walk.active == 0u) break;
            bool last;
            do {
                packet_walk(K, B, S);
                last = S.walk.sp == 0 && S.walk.lpos >= S.walk.nleaf * B.leaf;
                const int used = min(S.walk.nsurv, kPRound);
                last = last && used == S.walk.nsurv;
                const int groups = (used + 31) >> 5;
                for (int g = warp; g < groups; g += kPWarps) packet_test(K, B, S, g * 32, min(32, used - g * 32));
                __syncthreads();
                // the warps take the rays in turn: their work differs
                for (;;) {
                    int r = 0;
                    if (lane == 0) r = (int)atomicAdd(&S.next_ray, 1u);
                    r = __shfl_sync(kFull, r, 0);
                    if (r >= S.walk.n_rays) break;
                    if (S.walk.active >> r & 1u)
                        packet_ray<kMixed>(K, Lv, B, Bs, S, r, groups, S.list[warp], last);
                }
                __syncthreads();
                if (warp == 0) {  // the pieces that did not fit move up
                    const int left = S.walk.nsurv - used;
                    for (int k = lane; k < left; k += 32) S.surv[k] = S.surv[used + k];
                    __syncwarp();
                    if (lane == 0) {
                        S.walk.nsurv = left;
                        S.next_ray = 0;
                        if (O.tested) atomicAdd(O.tested, (unsigned long long)used * __popc(S.walk.active));
                    }
                }
                __syncthreads();
            } while (!last);
            // (a ray whose segments have ended may hold an attenuation that is no number, which segment_loop
            // never uses)
            if (warp == 0 && (S.walk.active >> lane & 1u)) {
                S.sum_r[lane] += S.attn_r[lane] * (float)S.acc_r[lane];
                S.sum_g[lane] += S.attn_g[lane] * (float)S.acc_g[lane];
                S.sum_b[lane] += S.attn_b[lane] * (float)S.acc_b[lane];
            }
            __syncthreads();
        }
        if (warp == 0 && S.ray_q[lane] >= 0)
            write_out(O, S.ray_q[lane], Rgb{S.sum_r[lane], S.sum_g[lane], S.sum_b[lane]}, S.cnt[lane], S.hash[lane], Q,
                      K.P.norm_bb1d);
        __syncthreads();
    }
}

// BB1D at cube1024: 2 blocks 215 ms, 3 185; 4 (with rounds of 512 pieces, an earlier version) 193 against 190
constexpr int kPBlocks = 3;

template <bool kMixed>
int blocks_per_sm()
{
    auto* f = k_bb1d_packet<kMixed, kPBlocks>;
    const int bytes = (int)sizeof(PacketShared);
    int nb = 0;
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, f, kPThreads, bytes);
    return nb > 0 ? nb : 1;
}

}  // namespace

int packet_max(int width, int height, int64_t n)
{
    return (int)std::min<int64_t>((int64_t)((width + 7) / 8) * ((height + 3) / 4), n);
}
int packet_slots(int packets, int resident) { return packets + (int)(2.f / kPacketShare) * resident + 2 * resident; }

void launch_packet_setup(const SegQueriesDev& Q, const uint32_t* keys, const int32_t* order, const uint32_t* cnt_pb2d,
                         int packets, int64_t n_pixels, const float* bbox, float piece_len, int resident,
                         const PacketsDev& P, cudaStream_t s)
{
    // the widest packet, in piece lengths
    constexpr float kPacketWidth = 4.f;
    k_packet_setup<<<(unsigned)((Q.n + 255) / 256), 256, 0, s>>>(Q, keys, order, cnt_pb2d, n_pixels, bbox,
                                                                 kPacketWidth * piece_len, P.range, P.weight, P.in_packet,
                                                                 P.totals);
    k_packet_items<<<(packets + 255) / 256, 256, 0, s>>>(P.weight, P.range, kPacketShare / (float)resident,
                                                         (unsigned)packet_slots(packets, resident), P.totals, P.key, P.item);
}

int bb1d_packet_blocks_per_sm(bool mixed) { return mixed ? blocks_per_sm<true>() : blocks_per_sm<false>(); }

void launch_bb1d_packet(const GatherConsts& K, const LightSoA& L, const BeamBVH& B, const BeamSoA& S,
                        const SegQueriesDev& Q, const Outputs& O, const int32_t* order, const PacketsDev& P,
                        const float* bbox, float piece_len, int grid, bool mixed, unsigned* work, cudaStream_t s)
{
    const int bytes = (int)sizeof(PacketShared);
    if (mixed)
        k_bb1d_packet<true, kPBlocks><<<grid, kPThreads, bytes, s>>>(
            K, L, B, S, Q, O, order, P.item_sorted, P.totals, bbox, piece_len, work);
    else
        k_bb1d_packet<false, kPBlocks><<<grid, kPThreads, bytes, s>>>(
            K, L, B, S, Q, O, order, P.item_sorted, P.totals, bbox, piece_len, work);
}

}  // namespace upbp
