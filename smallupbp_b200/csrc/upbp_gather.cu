// Gather kernels of the B200 estimator stage: one thread per recorded query.
//
//  * PB2D  : EmbreeBre::evalBre + breIntersectFuncHomogeneous2 (Bre/Bre.cxx:293-464, 812-964)
//  * BB1D  : PhotonBeamsEvaluator::evalBeamBeamEstimate + PhotonBeam::accumulate2
//            (Beams/PhBeams.cxx:177-324, Beams/PhotonBeam.hxx:386-607)
//  * PP3D  : HashGrid::Process + UPBP::RangeQuery::Process (Misc/HashGrid.hxx:129-188,
//            Renderers/UPBP.hxx:86-133)
// Candidate predicates use the reference operation order (upbp_device.cuh); the MIS weights
// walk the stored camera snapshot and light subpath exactly as Path/PathWeight.hxx does.
#include <cfloat>
#include <cstdint>

#include "upbp_contrib.cuh"

namespace upbp {

namespace {

// ----------------------------------------------------------------- kernels
template <bool kMixed>
__global__ void __launch_bounds__(256) k_gather_pb2d(const __grid_constant__ GatherConsts K, const LightSoA Lv,
                                                     const PhotonBVH B, const SegQueriesDev Q,
                                                     const upbp_mis* __restrict__ cam, const CamSum* __restrict__ cs,
                                                     const Outputs O, const int32_t* __restrict__ order)
{
    __shared__ DMedium media[UPBP_MAX_MEDIA];
    stage_media(K, media);
    const int64_t item = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (item >= Q.n) return;
    const int64_t q = order ? (int64_t)__ldg(&order[item]) : item;
    uint32_t cnt = 0;
    unsigned long long h = 0, tested = 0;
    Rgb res = rgb(0.f);
    if ((Q.flags[q] & UPBP_Q_PB2D) && (K.P.techniques & UPBP_PB2D) && B.n > 0) {
        SegCtx s;
        upbp_mis e_store;
        CamSum cs_store;
        init_seg_ctx<kMixed>(s, K, Q, cam, cs, q, &e_store, &cs_store);
        const V3 inv = v3(safe_inv(s.d.x), safe_inv(s.d.y), safe_inv(s.d.z));
        const float r2 = K.P.radius_pb2d * K.P.radius_pb2d;
        res = segment_loop(K, media, Q, q, s, [&](const DMedium& m) {
            Rgb acc = rgb(0.f);
            traverse(B.nodes, B.n_leaves, s.o, inv, s.dmin - K.eps, s.dmax + K.eps, [&](int leaf) {
                const int e = min(B.n, (leaf + 1) * B.leaf);
                for (int i = leaf * B.leaf; i < e; ++i) {
                    const float4 p = __ldg(&B.pos[i]);
                    ++tested;
                    float t, d2;
                    const float r2i = B.r2 ? __ldg(&B.r2[i]) : r2;
                    if (test_bre(s.o, s.d, s.dmin, s.dmax, v3(p.x, p.y, p.z), r2i, &t, &d2)) {
                        const int lv = __float_as_int(p.w);
                        ++cnt;
                        h += mix64((unsigned long long)lv);
                        acc = acc + pb2d_contrib<kMixed>(K, m, Lv, s, lv, t, d2, r2i);
                    }
                }
            });
            return acc;
        });
    }
    write_out(O, q, res, cnt, h, Q, K.P.norm_pb2d);
    if (O.tested) atomicAdd(O.tested, tested);
}

template <bool kMixed>
__global__ void __launch_bounds__(256) k_gather_bb1d(const __grid_constant__ GatherConsts K, const LightSoA Lv,
                                                     const BeamBVH B, const BeamSoA Bs, const SegQueriesDev Q,
                                                     const upbp_mis* __restrict__ cam, const CamSum* __restrict__ cs,
                                                     const Outputs O)
{
    __shared__ DMedium media[UPBP_MAX_MEDIA];
    stage_media(K, media);
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (q >= Q.n) return;
    uint32_t cnt = 0;
    unsigned long long h = 0, tested = 0;
    Rgb res = rgb(0.f);
    if ((Q.flags[q] & UPBP_Q_BB1D) && (K.P.techniques & UPBP_BB1D) && B.n > 0) {
        SegCtx s;
        upbp_mis e_store;
        CamSum cs_store;
        init_seg_ctx<kMixed>(s, K, Q, cam, cs, q, &e_store, &cs_store);
        const V3 inv = v3(safe_inv(s.d.x), safe_inv(s.d.y), safe_inv(s.d.z));
        res = segment_loop(K, media, Q, q, s, [&](const DMedium& m) {
            Rgb acc = rgb(0.f);
            const int mid = (int)(&m - media);
            traverse(B.nodes, B.n_leaves, s.o, inv, s.dmin - K.eps, s.dmax + K.eps, [&](int leaf) {
                const int e = min(B.n, (leaf + 1) * B.leaf);
                for (int i = leaf * B.leaf; i < e; ++i) {
                    const float4 pc = __ldg(&B.pc[i]);
                    if (__float_as_int(pc.w) != mid) continue;  // mMedium == medium (PhotonBeam.hxx:390)
                    const float4 pa = __ldg(&B.pa[i]);
                    const float4 pb = __ldg(&B.pb[i]);
                    ++tested;
                    float dist, sinT, t1, t2, bb, ee;
                    if (!test_beam_beam(s.o, s.d, s.dmin, s.dmax, v3(pa.x, pa.y, pa.z), v3(pb.x, pb.y, pb.z), 0.f, pa.w,
                                        pb.w, &dist, &sinT, &t1, &t2, &bb, &ee))
                        continue;
                    const int beam = __float_as_int(pc.z);
                    const float rs = beam_start_radius(Bs, &Bs.radius[beam]);
                    const float radius = beam_radius_at(Bs, beam, rs, t2);
                    if (radius < dist) continue;  // PhotonBeam.hxx:411-413
                    if (!piece_takes(s.o, s.d, s.dmin, s.dmax, v3(pa.x, pa.y, pa.z), v3(pb.x, pb.y, pb.z), pa.w, pc.x,
                                     pc.y, t1, bb, ee, dist, rs, Bs.rchange ? __ldg(&Bs.rchange[beam]) : 0.f,
                                     K.bb1d_extra))
                        continue;
                    ++cnt;
                    h += mix64((unsigned long long)beam);
                    acc = acc + bb1d_contrib<kMixed>(K, m, Lv, Bs, s, beam, v3(pa.x, pa.y, pa.z), v3(pb.x, pb.y, pb.z), radius,
                                                          dist, sinT, t1, t2);
                }
            });
            return acc;
        });
    }
    write_out(O, q, res, cnt, h, Q, K.P.norm_bb1d);
    if (O.tested) atomicAdd(O.tested, tested);
}

// Accepted candidates of one warp waiting for evaluation: the piece and its closest approach.
constexpr int kCandQueue = 64;
struct CandQueue {
    int piece[kCandQueue];
    float4 geo[kCandQueue];  // dist, sin(theta), t1 (query), t2 (beam)
    int near[kCandQueue];    // BB1D: pieces past the predicate's first check, waiting for the rest
};

// Per-warp scratch of the warp-cooperative gathers (shared memory).
struct WarpScratch {
    int* stack;
    int* leaves;
    CandQueue* cq;
    int lane;
    unsigned lt;  // lanes below this one
};

// BB1D of one query by one warp: the lanes test 32 beam pieces at a time; the accepted ones go to
// the warp's candidate queue, and whenever it holds 32 they are evaluated one per lane, so the
// contribution (transmittance, phase function, MIS weight) runs with every lane busy although
// only a fraction of the tested pieces is accepted.  Returns this lane's share of the result.
template <bool kMixed>
__device__ __forceinline__ Rgb bb1d_query_warp(const GatherConsts& K, const DMedium* media, const LightSoA& Lv,
                                               const BeamBVH& B, const BeamSoA& Bs, const SegQueriesDev& Q,
                                               int64_t q, SegCtx& s, V3 inv, const WarpScratch& ws,
                                               unsigned long long& cnt, unsigned long long& h,
                                               unsigned long long& tested, int* status)
{
    const int lane = ws.lane;
    const unsigned lt = ws.lt;
    CandQueue& cq = *ws.cq;
    const int leaf_shift = __ffs(B.leaf) - 1;
    unsigned cnt32 = 0, tested32 = 0;  // per query: below 2^32
    const Rgb res = segment_loop(K, media, Q, q, s, [&](const DMedium& m) {
        Rgb part = rgb(0.f);
        const int mid = (int)(&m - media);
        int qn = 0;  // entries in the candidate queue (warp-uniform)
        // evaluates queue entry e (one lane, one accepted candidate)
        auto eval = [&](int e) {
            const int i = cq.piece[e];
            const float4 g = cq.geo[e];
            const float4 pa = __ldg(&B.pa[i]);
            const float4 pb = __ldg(&B.pb[i]);
            const float4 pc = __ldg(&B.pc[i]);
            ++cnt32;
            h += mix64((unsigned long long)__float_as_int(pc.z));
            const int beam = __float_as_int(pc.z);
            if (kMixed) {
                const PiecePayload py = B.pay[i];
                const PairGeo pg{xdot3(s.d, v3(pb.x, pb.y, pb.z)), g.x * g.x, g.y, g.z, g.w};
                part = part + bb1d_contrib_packed<false>(K, m, s, py, pg, beam_radius_at(Bs, beam, py.lv.z, g.w));
            } else {
                part = part + bb1d_contrib<false>(K, m, Lv, Bs, s, beam, v3(pa.x, pa.y, pa.z), v3(pb.x, pb.y, pb.z),
                                                  beam_radius_at(Bs, beam, beam_start_radius(Bs, &Bs.radius[beam]), g.w), g.x, g.y,
                                                  g.z, g.w);
            }
        };
        // the rest of the predicate for one piece per lane (i < 0: none) that passed its first
        // check, with the ownership decision (in FP64 where the FP32 values cannot take it) and, in
        // mixed mode, the FP64 closest approach of near-parallel pairs; both run here rather than
        // in the evaluation, where the payload and the MIS inputs keep many more registers live.
        // Accepted candidates go to the candidate queue.
        auto full = [&](int i) {
            bool hit = false;
            float dist = 0.f, sinT = 0.f, t1 = 0.f, t2 = 0.f, bb = 0.f, ee = 0.f;
            if (i >= 0) {
                // the predicate reads only pa and pb; pc (piece interval, beam, medium) is loaded for
                // the pieces that pass it
                const float4 pa = __ldg(&B.pa[i]);
                const float4 pb = __ldg(&B.pb[i]);
                if (test_beam_beam(s.o, s.d, s.dmin, s.dmax, v3(pa.x, pa.y, pa.z), v3(pb.x, pb.y, pb.z), 0.f, pa.w,
                                   pb.w, &dist, &sinT, &t1, &t2, &bb, &ee)) {
                    const float4 pc = __ldg(&B.pc[i]);
                    if (__float_as_int(pc.w) == mid) {  // mMedium == medium (PhotonBeam.hxx:390)
                        // the radius test (PhotonBeam.hxx:411-413), then the reach rule and the owner
                        const int beam = __float_as_int(pc.z);
                        const float rs = beam_start_radius(Bs, kMixed ? &B.pay[i].lv.z : &Bs.radius[beam]);
                        const float rc = Bs.rchange ? __ldg(&Bs.rchange[beam]) : 0.f;
                        const float radius = beam_radius_at(Bs, beam, rs, t2);
                        hit = !(radius < dist);
                        if (hit) {
                            const int own = piece_takes_fast(s.o, s.d, s.dmin, s.dmax, v3(pa.x, pa.y, pa.z), pa.w,
                                                             pc.x, pc.y, t1, bb, ee, dist, rs, rc, K.bb1d_extra);
                            // the FP32 values cannot decide: the FP64 closest points of the segments
                            hit = own >= 0 ? own == 1
                                           : piece_takes_f64(s.o, s.d, s.dmin, s.dmax, v3(pa.x, pa.y, pa.z),
                                                             v3(pb.x, pb.y, pb.z), pa.w, pc.x, pc.y, rs, rc,
                                                             K.bb1d_extra);
                        }
                        if (kMixed && hit) {
                            // near-parallel lines, 1 - (d1.d2)^2 small: the FP32 solve of
                            // PhotonBeam.hxx:253-293 cancels, so the contribution gets the FP64
                            // closest approach (the candidate decision above stays FP32)
                            const float c = s.d.x * pb.x + s.d.y * pb.y + s.d.z * pb.z;
                            if (1.f - c * c < 1e-2f)
                                closest_approach_f64(s.o, s.d, v3(pa.x, pa.y, pa.z), v3(pb.x, pb.y, pb.z), dist,
                                                     sinT, t1, t2);
                        }
                    }
                }
            }
            const unsigned vote = __ballot_sync(kFull, hit);
            if (vote == 0u) return;
            if (hit) {
                const int pos = qn + __popc(vote & lt);
                cq.piece[pos] = i;
                cq.geo[pos] = make_float4(dist, sinT, t1, t2);
            }
            qn += __popc(vote);
            __syncwarp();
            if (qn >= 32) {  // the newest 32 entries, one per lane
                eval(qn - 32 + lane);
                qn -= 32;
                __syncwarp();
            }
        };
        // about a third of the tested pieces pass the predicate's first check (the distance of the
        // lines); they are queued and the rest of the predicate runs 32 at a time
        int pn = 0;  // entries in the near queue (warp-uniform)
        const bool ok = warp_traverse(B.nodes, B.n_leaves, B.n, leaf_shift, s.o, inv, s.dmin - K.eps, s.dmax + K.eps,
                                      ws.stack, ws.leaves, lane, [&](int i) {
            bool near = false;
            if (i >= 0) {
                const float4 pa = __ldg(&B.pa[i]);
                const float4 pb = __ldg(&B.pb[i]);
                ++tested32;
                near = beam_beam_near(s.o, s.d, v3(pa.x, pa.y, pa.z), v3(pb.x, pb.y, pb.z), pb.w);
            }
            const unsigned vote = __ballot_sync(kFull, near);
            if (vote == 0u) return;
            if (near) cq.near[pn + __popc(vote & lt)] = i;
            pn += __popc(vote);
            __syncwarp();
            if (pn >= 32) {
                full(cq.near[pn - 32 + lane]);
                pn -= 32;
                __syncwarp();
            }
        });
        if (pn > 0) {
            full(lane < pn ? cq.near[lane] : -1);
            __syncwarp();
        }
        if (lane < qn) eval(lane);
        __syncwarp();
        if (!ok && lane == 0) atomicOr(status, 1);
        return part;
    });
    cnt += cnt32;
    tested += tested32;
    return res;
}

// PB2D of one query by one warp over the photon LBVH, with the same candidate queue.
template <bool kMixed>
__device__ __forceinline__ Rgb pb2d_query_warp(const GatherConsts& K, const DMedium* media, const LightSoA& Lv,
                                               const PhotonBVH& P, const SegQueriesDev& Q, int64_t q, SegCtx& s,
                                               V3 inv, const WarpScratch& ws, unsigned long long& cnt,
                                               unsigned long long& h, unsigned long long& tested, int* status)
{
    const int lane = ws.lane;
    const unsigned lt = ws.lt;
    CandQueue& cq = *ws.cq;
    const int leaf_shift = __ffs(P.leaf) - 1;
    const float r2 = K.P.radius_pb2d * K.P.radius_pb2d;
    return segment_loop(K, media, Q, q, s, [&](const DMedium& m) {
        Rgb part = rgb(0.f);
        int qn = 0;
        auto eval = [&](int e) {
            const float4 g = cq.geo[e];
            part = part + pb2d_contrib<kMixed>(K, m, Lv, s, cq.piece[e], g.x, g.y, g.z);
        };
        const bool ok = warp_traverse(P.nodes, P.n_leaves, P.n, leaf_shift, s.o, inv, s.dmin - K.eps, s.dmax + K.eps,
                                      ws.stack, ws.leaves, lane, [&](int i) {
            bool hit = false;
            float t = 0.f, d2 = 0.f, r2i = r2;
            int lv = 0;
            if (i >= 0) {
                const float4 p = __ldg(&P.pos[i]);
                ++tested;
                if (P.r2) r2i = __ldg(&P.r2[i]);
                if (test_bre(s.o, s.d, s.dmin, s.dmax, v3(p.x, p.y, p.z), r2i, &t, &d2)) {
                    lv = __float_as_int(p.w);
                    hit = true;
                    ++cnt;
                    h += mix64((unsigned long long)lv);
                }
            }
            const unsigned vote = __ballot_sync(kFull, hit);
            if (vote == 0u) return;
            if (hit) {
                const int pos = qn + __popc(vote & lt);
                cq.piece[pos] = lv;
                cq.geo[pos] = make_float4(t, d2, r2i, 0.f);
            }
            qn += __popc(vote);
            __syncwarp();
            if (qn >= 32) {
                eval(qn - 32 + lane);
                qn -= 32;
                __syncwarp();
            }
        });
        if (lane < qn) eval(lane);
        __syncwarp();
        if (!ok && lane == 0) atomicOr(status, 1);
        return part;
    });
}

// BB1D, warp per query, persistent: warps draw query indices (in Morton order of the query
// midpoints) from an atomic counter.  elsewhere: how many queries at the end of the order the packet
// gather evaluates (NULL: none).  The launch may overlap that gather's, whose results nothing here reads; every
// block waits for its end, so that what follows in the stream follows both.
template <bool kMixed, int kWarps, int kMinBlocks>
__global__ void __launch_bounds__(kWarps * 32, kMinBlocks) k_bb1d_warp(const __grid_constant__ GatherConsts K, const LightSoA Lv,
                                                          const BeamBVH B, const BeamSoA Bs, const SegQueriesDev Q,
                                                          const upbp_mis* __restrict__ cam,
                                                          const CamSum* __restrict__ cs, const Outputs O,
                                                          unsigned int* __restrict__ work, int* __restrict__ status,
                                                          const int32_t* __restrict__ order,
                                                          const unsigned* __restrict__ elsewhere)
{
    __shared__ DMedium media[UPBP_MAX_MEDIA];
    __shared__ int s_stack[kWarps][kWarpStack];
    __shared__ int s_leaves[kWarps][kWarpLeaves];
    __shared__ CandQueue s_queue[kWarps];
    __shared__ upbp_mis s_e[kWarps];
    __shared__ CamSum s_cs[kWarps];
    stage_media(K, media);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const WarpScratch ws{s_stack[warp], s_leaves[warp], &s_queue[warp], lane, (1u << lane) - 1u};
    const int64_t n_items = Q.n - (elsewhere ? (int64_t)*elsewhere : 0);
    for (;;) {
        unsigned qq = 0;
        if (lane == 0) qq = atomicAdd(work, 1u);
        const int64_t item = (int64_t)__shfl_sync(kFull, qq, 0);
        if (item >= n_items) break;
        const int64_t q = order ? (int64_t)__ldg(&order[item]) : item;
        Rgb acc = rgb(0.f);
        unsigned long long cnt = 0, h = 0, tested = 0;
        if ((Q.flags[q] & UPBP_Q_BB1D) && (K.P.techniques & UPBP_BB1D) && B.n > 0) {
            SegCtx s;
            init_seg_ctx<kMixed>(s, K, Q, cam, cs, q, &s_e[warp], &s_cs[warp], lane == 0);
            __syncwarp();
            const V3 inv = v3(safe_inv(s.d.x), safe_inv(s.d.y), safe_inv(s.d.z));
            acc = bb1d_query_warp<kMixed>(K, media, Lv, B, Bs, Q, q, s, inv, ws, cnt, h, tested, status);
        }
        const float r = warp_sum(acc.r), g = warp_sum(acc.g), b = warp_sum(acc.b);
        cnt = warp_sum_u64(cnt);
        h = warp_sum_u64(h);
        tested = warp_sum_u64(tested);
        if (lane == 0) {
            O.rgb[3 * q + 0] = r;
            O.rgb[3 * q + 1] = g;
            O.rgb[3 * q + 2] = b;
            if (O.count) O.count[q] = (uint32_t)cnt;
            if (O.hash) O.hash[q] = h;
            const Rgb thr{Q.throughput[3 * q], Q.throughput[3 * q + 1], Q.throughput[3 * q + 2]};
            splat(O.image, Q.pixel[q], thr * K.P.norm_bb1d * Rgb{r, g, b});
            if (O.tested) atomicAdd(O.tested, tested);
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// PB2D, warp per query, persistent (the BB1D kernel's scheme over the photon LBVH): the lanes
// test 32 photons at a time and evaluate the accepted ones 32 at a time from the candidate queue.
template <bool kMixed, int kWarps, int kMinBlocks>
__global__ void __launch_bounds__(kWarps * 32, kMinBlocks) k_pb2d_warp(const __grid_constant__ GatherConsts K,
                                                                     const LightSoA Lv, const PhotonBVH P,
                                                                     const SegQueriesDev Q,
                                                                     const upbp_mis* __restrict__ cam,
                                                                     const CamSum* __restrict__ cs, const Outputs O,
                                                                     unsigned int* __restrict__ work,
                                                                     int* __restrict__ status,
                                                                     const int32_t* __restrict__ order)
{
    __shared__ DMedium media[UPBP_MAX_MEDIA];
    __shared__ int s_stack[kWarps][kWarpStack];
    __shared__ int s_leaves[kWarps][kWarpLeaves];
    __shared__ CandQueue s_queue[kWarps];
    __shared__ upbp_mis s_e[kWarps];
    __shared__ CamSum s_cs[kWarps];
    stage_media(K, media);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const WarpScratch ws{s_stack[warp], s_leaves[warp], &s_queue[warp], lane, (1u << lane) - 1u};
    for (;;) {
        unsigned qq = 0;
        if (lane == 0) qq = atomicAdd(work, 1u);
        const int64_t item = (int64_t)__shfl_sync(kFull, qq, 0);
        if (item >= Q.n) break;
        const int64_t q = order ? (int64_t)__ldg(&order[item]) : item;
        Rgb acc = rgb(0.f);
        unsigned long long cnt = 0, h = 0, tested = 0;
        if ((Q.flags[q] & UPBP_Q_PB2D) && (K.P.techniques & UPBP_PB2D) && P.n > 0) {
            SegCtx s;
            init_seg_ctx<kMixed>(s, K, Q, cam, cs, q, &s_e[warp], &s_cs[warp], lane == 0);
            __syncwarp();
            const V3 inv = v3(safe_inv(s.d.x), safe_inv(s.d.y), safe_inv(s.d.z));
            acc = pb2d_query_warp<kMixed>(K, media, Lv, P, Q, q, s, inv, ws, cnt, h, tested, status);
        }
        const float r = warp_sum(acc.r), g = warp_sum(acc.g), b = warp_sum(acc.b);
        cnt = warp_sum_u64(cnt);
        h = warp_sum_u64(h);
        tested = warp_sum_u64(tested);
        if (lane == 0) {
            O.rgb[3 * q + 0] = r;
            O.rgb[3 * q + 1] = g;
            O.rgb[3 * q + 2] = b;
            if (O.count) O.count[q] = (uint32_t)cnt;
            if (O.hash) O.hash[q] = h;
            const Rgb thr{Q.throughput[3 * q], Q.throughput[3 * q + 1], Q.throughput[3 * q + 2]};
            splat(O.image, Q.pixel[q], thr * K.P.norm_pb2d * Rgb{r, g, b});
            if (O.tested) atomicAdd(O.tested, tested);
        }
    }
}

// All camera segments of an iteration in one persistent work-queue kernel: a warp takes the next
// query (Morton order) and evaluates both segment estimators for it, PB2D over the photon LBVH
// and BB1D over the beam-piece LBVH, with one camera context and one splat per query.
template <bool kMixed, int kWarps, int kMinBlocks>
__global__ void __launch_bounds__(kWarps * 32, kMinBlocks) k_segments_warp(
    const __grid_constant__ GatherConsts K, const LightSoA Lv, const PhotonBVH P, const BeamBVH B, const BeamSoA Bs,
    const SegQueriesDev Q, const upbp_mis* __restrict__ cam, const CamSum* __restrict__ cs, const Outputs Opb,
    const Outputs Obb, unsigned int* __restrict__ work, int* __restrict__ status, const int32_t* __restrict__ order)
{
    __shared__ DMedium media[UPBP_MAX_MEDIA];
    __shared__ int s_stack[kWarps][kWarpStack];
    __shared__ int s_leaves[kWarps][kWarpLeaves];
    __shared__ CandQueue s_queue[kWarps];
    __shared__ upbp_mis s_e[kWarps];
    __shared__ CamSum s_cs[kWarps];
    stage_media(K, media);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const WarpScratch ws{s_stack[warp], s_leaves[warp], &s_queue[warp], lane, (1u << lane) - 1u};
    for (;;) {
        unsigned qq = 0;
        if (lane == 0) qq = atomicAdd(work, 1u);
        const int64_t item = (int64_t)__shfl_sync(kFull, qq, 0);
        if (item >= Q.n) break;
        const int64_t q = order ? (int64_t)__ldg(&order[item]) : item;
        const uint32_t qf = Q.flags[q];
        const bool do_pb = (qf & UPBP_Q_PB2D) && (K.P.techniques & UPBP_PB2D) && P.n > 0;
        const bool do_bb = (qf & UPBP_Q_BB1D) && (K.P.techniques & UPBP_BB1D) && B.n > 0;
        Rgb apb = rgb(0.f), abb = rgb(0.f);
        unsigned long long cpb = 0, hpb = 0, tpb = 0, cbb = 0, hbb = 0, tbb = 0;
        if (do_pb || do_bb) {
            SegCtx s;
            init_seg_ctx<kMixed>(s, K, Q, cam, cs, q, &s_e[warp], &s_cs[warp], lane == 0);
            __syncwarp();
            const V3 inv = v3(safe_inv(s.d.x), safe_inv(s.d.y), safe_inv(s.d.z));
            if (do_pb) apb = pb2d_query_warp<kMixed>(K, media, Lv, P, Q, q, s, inv, ws, cpb, hpb, tpb, status);
            if (do_bb) abb = bb1d_query_warp<kMixed>(K, media, Lv, B, Bs, Q, q, s, inv, ws, cbb, hbb, tbb, status);
        }
        const Rgb vpb{warp_sum(apb.r), warp_sum(apb.g), warp_sum(apb.b)};
        const Rgb vbb{warp_sum(abb.r), warp_sum(abb.g), warp_sum(abb.b)};
        cpb = warp_sum_u64(cpb);
        hpb = warp_sum_u64(hpb);
        tpb = warp_sum_u64(tpb);
        cbb = warp_sum_u64(cbb);
        hbb = warp_sum_u64(hbb);
        tbb = warp_sum_u64(tbb);
        if (lane == 0) {
            Opb.rgb[3 * q + 0] = vpb.r;
            Opb.rgb[3 * q + 1] = vpb.g;
            Opb.rgb[3 * q + 2] = vpb.b;
            Obb.rgb[3 * q + 0] = vbb.r;
            Obb.rgb[3 * q + 1] = vbb.g;
            Obb.rgb[3 * q + 2] = vbb.b;
            if (Opb.count) Opb.count[q] = (uint32_t)cpb;
            if (Opb.hash) Opb.hash[q] = hpb;
            if (Obb.count) Obb.count[q] = (uint32_t)cbb;
            if (Obb.hash) Obb.hash[q] = hbb;
            const Rgb thr{Q.throughput[3 * q], Q.throughput[3 * q + 1], Q.throughput[3 * q + 2]};
            splat(Obb.image, Q.pixel[q], thr * (vpb * K.P.norm_pb2d + vbb * K.P.norm_bb1d));
            if (Opb.tested) atomicAdd(Opb.tested, tpb);
            if (Obb.tested) atomicAdd(Obb.tested, tbb);
        }
    }
}

// PP3D, 8 lanes per query: lane j looks up cell j of the 8 hashed cells, and the lanes then take the
// cells' photons in turn.  A query tests about 8 photons (cube1024: 7.5) through a chain of dependent
// loads (cell, photon, light vertex, MIS record), so with one thread per query the launch lasted as long
// as the longest run of photons: cube1024 0.477 -> 0.141 ms (plain), boxes3 1.17 -> 0.52 ms, 940 queries over
// 41 k photons 60 -> 19 us.
template <bool kMixed>
__global__ void __launch_bounds__(256) k_gather_pp3d(const __grid_constant__ GatherConsts K, const LightSoA Lv,
                                                     const HashGridDev G, const PointQueriesDev Q,
                                                     const upbp_mis* __restrict__ cam, const CamSum* __restrict__ cs,
                                                     const Outputs O)
{
    constexpr int kLanes = 8;
    __shared__ DMedium media[UPBP_MAX_MEDIA];
    stage_media(K, media);
    const int64_t q = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kLanes;
    const int j = threadIdx.x % kLanes;
    const bool live = q < Q.n;
    const upbp_params& P = K.P;
    uint32_t cnt = 0, tested = 0;
    unsigned long long h = 0;
    Rgb res = rgb(0.f);
    V3 qp{0.f, 0.f, 0.f}, dmin{0.f, 0.f, 0.f};
    bool inside = live && (P.techniques & UPBP_PP3D) && G.n > 0;
    if (inside) {
        qp = v3(Q.position[3 * q], Q.position[3 * q + 1], Q.position[3 * q + 2]);
        dmin = xsub3(qp, v3(G.bbox_min[0], G.bbox_min[1], G.bbox_min[2]));
        const V3 dmax = xsub3(v3(G.bbox_max[0], G.bbox_max[1], G.bbox_max[2]), qp);
        inside = !(dmin.x < 0.f || dmin.y < 0.f || dmin.z < 0.f || dmax.x < 0.f || dmax.y < 0.f || dmax.z < 0.f);
    }
    // the lane's cell: its photons are items [before, before + mine) of the query's
    int begin = 0, mine = 0;
    if (inside) {
        const V3 cell = v3(xmul(G.inv_cell, dmin.x), xmul(G.inv_cell, dmin.y), xmul(G.inv_cell, dmin.z));
        const V3 cf = v3(floorf(cell.x), floorf(cell.y), floorf(cell.z));
        const int px = (int)cf.x, py = (int)cf.y, pz = (int)cf.z;
        const int cx = (j & 4) ? px + (xsub(cell.x, cf.x) < 0.5f ? -1 : 1) : px;
        const int cy = (j & 2) ? py + (xsub(cell.y, cf.y) < 0.5f ? -1 : 1) : py;
        const int cz = (j & 1) ? pz + (xsub(cell.z, cf.z) < 0.5f ? -1 : 1) : pz;
        const uint32_t c = hash_cell(cx, cy, cz, G.cells);
        begin = __ldg(&G.start[c]);
        mine = __ldg(&G.end[c]) - begin;
    }
    int upto = mine;
#pragma unroll
    for (int d = 1; d < kLanes; d <<= 1) {
        const int v = __shfl_up_sync(kFull, upto, d, kLanes);
        if (j >= d) upto += v;
    }
    const int total = __shfl_sync(kFull, upto, kLanes - 1, kLanes);
    const int first = begin - (upto - mine);  // item k of this cell is photon first + k
    const int mid = inside ? Q.medium_id[q] : 0;
    const DMedium& m = media[mid];
    const int L = inside ? Q.path_length[q] : 0;
    const CamSnap camv{cam + (inside ? Q.cam_mis_begin[q] : 0)};
    const bool scat_pos = !(m.ss[0] <= 0.f && m.ss[1] <= 0.f && m.ss[2] <= 0.f);
    const int rounds = (__reduce_max_sync(kFull, total) + kLanes - 1) / kLanes;
    for (int it = 0; it < rounds; ++it) {
        const int k = it * kLanes + j;
        int c = 0;  // the cell of item k: the first whose items end beyond k
#pragma unroll
        for (int d = kLanes / 2; d > 0; d >>= 1)
            if (__shfl_sync(kFull, upto, c + d - 1, kLanes) <= k) c += d;
        const int i = __shfl_sync(kFull, first, c, kLanes) + k;
        if (k >= total) continue;
        const float4 p = __ldg(&G.pos[i]);
        ++tested;
        const V3 dd = xsub3(qp, v3(p.x, p.y, p.z));
        if (!(xdot3(dd, dd) <= G.r2)) continue;
        const int lv = __float_as_int(p.w);
        ++cnt;
        h += mix64((unsigned long long)lv);
        // UPBP::RangeQuery::Process (UPBP.hxx:86-133)
        const int4 info = __ldg(&Lv.info[lv]);
        if (!(info.z & UPBP_LV_CONNECTABLE)) continue;
        const int pl = info.y;
        if ((uint32_t)(pl + L) > P.max_path_length || (uint32_t)(pl + L) < P.min_path_length) continue;
        if (!scat_pos) continue;
        const float4 ld = __ldg(&Lv.dir[lv]);
        const V3 cfix = v3(Q.dir_fix[3 * q], Q.dir_fix[3 * q + 1], Q.dir_fix[3 * q + 2]);
        float sinT;
        const float phase = hg_pdf(cfix, v3(ld.x, ld.y, ld.z), m.g, &sinT);
        const Rgb factor = Rgb{m.ss[0], m.ss[1], m.ss[2]} * phase;
        if (rgb_black_or_neg(factor)) continue;
        const float dirPdf = phase * m.cont;
        const float revPdf = phase * __ldg(&Lv.pos[lv]).w;
        const upbp_mis lvm = load_mis(Lv.mis + lv);
        const float mwfInv = 1.0f / lvm.pp3d_factor;
        float wCamera, wLight;
        if (kMixed) {
            const upbp_mis eL = load_mis(camv.snap + L);
            upbp_mis eL1{};
            if (L >= 2) eL1 = load_mis(camv.snap + L - 1);
            wCamera = camera_weight_fast(L, eL, mwfInv, sinT, lvm.ray_sample_pdf_inv, lvm.ray_sample_pdfs_ratio, revPdf,
                                         eL1, eL1.ray_sample_rev_pdf_inv, cs[q], P.techniques, P.query_beam_type,
                                         P.photon_beam_type);
            const LightSum ls = Lv.sums[lv];
            wLight = mwfInv * ((float)ls.a + dirPdf * (float)ls.c);
        } else {
            wCamera = camera_path_weight(L, mwfInv, sinT, lvm.ray_sample_pdf_inv, lvm.ray_sample_pdfs_ratio, revPdf,
                                         P.query_beam_type, P.photon_beam_type, P.techniques, camv);
            const LightView lview{Lv.mis, -1, 0.f};
            wLight = light_path_weight(info.x, pl, mwfInv, 0.f, 0.f, 0.f, dirPdf, UPBP_PP3D, P.query_beam_type,
                                       P.photon_beam_type, P.techniques, Lv.path_ends, lview, nullptr);
        }
        const float w = 1.f / (wLight + wCamera);
        const float4 th = __ldg(&Lv.thr[lv]);
        res = res + w * (factor * Rgb{th.x, th.y, th.z});
    }
#pragma unroll
    for (int d = kLanes / 2; d > 0; d >>= 1) {
        res.r += __shfl_xor_sync(kFull, res.r, d);
        res.g += __shfl_xor_sync(kFull, res.g, d);
        res.b += __shfl_xor_sync(kFull, res.b, d);
        cnt += __shfl_xor_sync(kFull, cnt, d);
        h += __shfl_xor_sync(kFull, h, d);
    }
    if (O.tested) {
        tested = __reduce_add_sync(kFull, tested);
        if ((threadIdx.x & 31) == 0 && tested) atomicAdd(O.tested, (unsigned long long)tested);
    }
    if (!live || j != 0) return;
    O.rgb[3 * q + 0] = res.r;
    O.rgb[3 * q + 1] = res.g;
    O.rgb[3 * q + 2] = res.b;
    if (O.count) O.count[q] = cnt;
    if (O.hash) O.hash[q] = h;
    const Rgb thr{Q.throughput[3 * q], Q.throughput[3 * q + 1], Q.throughput[3 * q + 2]};
    splat(O.image, Q.pixel[q], thr * P.norm_pp3d * res);
}

// B-P2D (extension; the reference has no beam x point estimator): photon beams queried at the
// camera medium vertices with a 2-D kernel, MIS weight 1.  Candidate: testIntersectionBre with
// the beam as the ray and the query point as the photon; the piece containing the foot point
// takes it.  Value: beam throughput x transmittance to the foot point (divided by the free-flight
// pdf for SHORT beams) x sigma_s x HG phase x (1 - d^2/r^2) / (pi r^2 / 2).
// B-P2D contribution of one accepted (point, beam) pair: beam throughput x transmittance to the
// foot point t (divided by the free-flight pdf for SHORT beams) x sigma_s x HG x the 2-D kernel.
__device__ __forceinline__ Rgb bp2d_contrib(const DMedium& m, const BeamSoA& Bs, int beam, V3 cfix, V3 bdir, float t,
                                            float d2, float r2)
{
    const float4 bthr = __ldg(&Bs.thr[beam]);
    Rgb att = eval_att(m, t);
    const float pfd = comp(att, m.min_idx);
    if ((uint32_t)__float_as_int(bthr.w) & UPBP_SHORT_BEAM) att = att / pfd;
    if (!rgb_positive(att)) return rgb(0.f);
    float sinT;
    const float phase = hg_pdf(cfix, neg3(bdir), m.g, &sinT);
    if (phase <= 0.f) return rgb(0.f);
    const float kernel = (1.f - d2 / r2) / (r2 * UPBP_PI_F * 0.5f);
    if (!is_pos(kernel)) return rgb(0.f);
    const Rgb ss{m.ss[0], m.ss[1], m.ss[2]};
    return Rgb{bthr.x, bthr.y, bthr.z} * att * ss * (phase * kernel);
}

// B-P2D, warp per point query, persistent: the lanes test 32 beam pieces at a time (the zero-length
// ray at the point makes the slab test a point-in-box test); accepted pairs go to the candidate
// queue and are evaluated 32 at a time.
template <int kWarps, int kMinBlocks>
__global__ void __launch_bounds__(kWarps * 32, kMinBlocks) k_bp2d_warp(const __grid_constant__ GatherConsts K,
                                                                     const BeamBVH B, const BeamSoA Bs,
                                                                     const PointQueriesDev Q, const Outputs O,
                                                                     unsigned int* __restrict__ work,
                                                                     int* __restrict__ status)
{
    __shared__ DMedium media[UPBP_MAX_MEDIA];
    __shared__ int s_stack[kWarps][kWarpStack];
    __shared__ int s_leaves[kWarps][kWarpLeaves];
    __shared__ CandQueue s_queue[kWarps];
    stage_media(K, media);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    int* stack = s_stack[warp];
    int* leaves = s_leaves[warp];
    CandQueue& cq = s_queue[warp];
    const int leaf_shift = __ffs(B.leaf) - 1;
    for (;;) {
        unsigned qq = 0;
        if (lane == 0) qq = atomicAdd(work, 1u);
        const int64_t q = (int64_t)__shfl_sync(kFull, qq, 0);
        if (q >= Q.n) break;
        Rgb part = rgb(0.f);
        unsigned long long cnt = 0, h = 0, tested = 0;
        const int mid = Q.medium_id[q];
        const DMedium& m = media[mid];
        if ((K.P.techniques & UPBP_BP2D) && m.has_scat && B.n > 0) {
            const V3 x = v3(Q.position[3 * q], Q.position[3 * q + 1], Q.position[3 * q + 2]);
            const V3 cfix = v3(Q.dir_fix[3 * q], Q.dir_fix[3 * q + 1], Q.dir_fix[3 * q + 2]);
            int qn = 0;
            auto eval = [&](int e) {
                const int i = cq.piece[e];
                const float4 g = cq.geo[e];  // t, d^2, r^2, -
                const float4 pb = __ldg(&B.pb[i]);
                const float4 pc = __ldg(&B.pc[i]);
                part = part + bp2d_contrib(m, Bs, __float_as_int(pc.z), cfix, v3(pb.x, pb.y, pb.z), g.x, g.y, g.z);
            };
            const bool ok = warp_traverse(B.nodes, B.n_leaves, B.n, leaf_shift, x, v3(1.f, 1.f, 1.f), 0.f, 0.f, stack,
                                          leaves, lane, [&](int i) {
                bool hit = false;
                float t = 0.f, d2 = 0.f, r2 = 0.f;
                if (i >= 0) {
                    const float4 pc = __ldg(&B.pc[i]);
                    if (__float_as_int(pc.w) == mid) {
                        const float4 pa = __ldg(&B.pa[i]);
                        const float4 pb = __ldg(&B.pb[i]);
                        ++tested;
                        // bound: the beam's largest radius^2; then the radius at the foot point
                        if (test_bre(v3(pa.x, pa.y, pa.z), v3(pb.x, pb.y, pb.z), 0.f, pa.w, x, pb.w, &t, &d2) &&
                            t >= pc.x && t < pc.y) {  // the piece containing the foot point
                            const int beam = __float_as_int(pc.z);
                            const float rt = beam_radius_at(Bs, beam, beam_start_radius(Bs, &Bs.radius[beam]), t);
                            r2 = rt * rt;
                            if (!(Bs.rchange && d2 > r2)) {
                                hit = true;
                                ++cnt;
                                h += mix64((unsigned long long)beam);
                            }
                        }
                    }
                }
                const unsigned vote = __ballot_sync(kFull, hit);
                if (vote == 0u) return;
                if (hit) {
                    const int pos = qn + __popc(vote & lt);
                    cq.piece[pos] = i;
                    cq.geo[pos] = make_float4(t, d2, r2, 0.f);
                }
                qn += __popc(vote);
                __syncwarp();
                if (qn >= 32) {
                    eval(qn - 32 + lane);
                    qn -= 32;
                    __syncwarp();
                }
            });
            if (lane < qn) eval(lane);
            __syncwarp();
            if (!ok && lane == 0) atomicOr(status, 1);
        }
        const float r = warp_sum(part.r), g = warp_sum(part.g), b = warp_sum(part.b);
        cnt = warp_sum_u64(cnt);
        h = warp_sum_u64(h);
        tested = warp_sum_u64(tested);
        if (lane == 0) {
            O.rgb[3 * q + 0] = r;
            O.rgb[3 * q + 1] = g;
            O.rgb[3 * q + 2] = b;
            if (O.count) O.count[q] = (uint32_t)cnt;
            if (O.hash) O.hash[q] = h;
            const Rgb thr{Q.throughput[3 * q], Q.throughput[3 * q + 1], Q.throughput[3 * q + 2]};
            splat(O.image, Q.pixel[q], thr * K.P.norm_bb1d * Rgb{r, g, b});
            if (O.tested) atomicAdd(O.tested, tested);
        }
    }
}

__global__ void __launch_bounds__(256) k_gather_bp2d(const __grid_constant__ GatherConsts K, const BeamBVH B,
                                                     const BeamSoA Bs, const PointQueriesDev Q, const Outputs O)
{
    __shared__ DMedium media[UPBP_MAX_MEDIA];
    stage_media(K, media);
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (q >= Q.n) return;
    uint32_t cnt = 0;
    unsigned long long h = 0, tested = 0;
    Rgb res = rgb(0.f);
    const V3 x = v3(Q.position[3 * q], Q.position[3 * q + 1], Q.position[3 * q + 2]);
    const int mid = Q.medium_id[q];
    const DMedium& m = media[mid];
    if ((K.P.techniques & UPBP_BP2D) && m.has_scat && B.n > 0) {
        const V3 cfix = v3(Q.dir_fix[3 * q], Q.dir_fix[3 * q + 1], Q.dir_fix[3 * q + 2]);
        // a zero-length ray at x: the slab test becomes point-in-box
        traverse(B.nodes, B.n_leaves, x, v3(1.f, 1.f, 1.f), 0.f, 0.f, [&](int leaf) {
            const int e = min(B.n, (leaf + 1) * B.leaf);
            for (int i = leaf * B.leaf; i < e; ++i) {
                const float4 pc = __ldg(&B.pc[i]);
                if (__float_as_int(pc.w) != mid) continue;
                const float4 pa = __ldg(&B.pa[i]);
                const float4 pb = __ldg(&B.pb[i]);
                ++tested;
                float t, d2;
                // bound: the beam's largest radius^2; then the radius at the foot point
                if (!test_bre(v3(pa.x, pa.y, pa.z), v3(pb.x, pb.y, pb.z), 0.f, pa.w, x, pb.w, &t, &d2)) continue;
                if (!(t >= pc.x && t < pc.y)) continue;  // the piece containing the foot point
                const int beam = __float_as_int(pc.z);
                const float rt = beam_radius_at(Bs, beam, beam_start_radius(Bs, &Bs.radius[beam]), t), r2 = rt * rt;
                if (Bs.rchange && d2 > r2) continue;
                ++cnt;
                h += mix64((unsigned long long)beam);
                res = res + bp2d_contrib(m, Bs, beam, cfix, v3(pb.x, pb.y, pb.z), t, d2, r2);
            }
        });
    }
    O.rgb[3 * q + 0] = res.r;
    O.rgb[3 * q + 1] = res.g;
    O.rgb[3 * q + 2] = res.b;
    if (O.count) O.count[q] = cnt;
    if (O.hash) O.hash[q] = h;
    const Rgb thr{Q.throughput[3 * q], Q.throughput[3 * q + 1], Q.throughput[3 * q + 2]};
    splat(O.image, Q.pixel[q], thr * K.P.norm_bb1d * res);
    if (O.tested) atomicAdd(O.tested, tested);
}

// ----------------------------------------------------------------- BB1D over the beam grid
// SSE min_ps / max_ps: the second operand unless the first compares below / above it
__device__ __forceinline__ float sse_min(float a, float b) { return a < b ? a : b; }
__device__ __forceinline__ float sse_max(float a, float b) { return a > b ? a : b; }
__device__ __forceinline__ float pick3(int k, float a, float b, float c) { return k == 0 ? a : (k == 1 ? b : c); }

// Grid::intersect (Grid.hxx:322-398): the DDA walk of one segment [mint, maxt] of the query ray
// through the reference's grid, with the reference's float operations (the box test of
// BoundingBox3::intersect, Structs/BoundingBox.hxx:218-272, with its SSE operand order, which
// turns the NaN of a zero direction component into an unbounded slab).  visit(cell, cell_mint,
// cell_maxt) for every visited cell, in order; the walk leaves the grid after at most
// res0 + res1 + res2 cells.
template <class Visit>
__device__ __forceinline__ void grid_walk(const GridHeader& h, V3 o, V3 d, float mint, float maxt, Visit&& visit)
{
    const float ix = __fdiv_rn(1.f, d.x), iy = __fdiv_rn(1.f, d.y), iz = __fdiv_rn(1.f, d.z);
    float lmax = 0.f, lmin = 0.f;
    for (int k = 0; k < 3; ++k) {
        const float ok = pick3(k, o.x, o.y, o.z), ik = pick3(k, ix, iy, iz);
        const float l1 = __fmul_rn(__fsub_rn(h.lo[k], ok), ik);
        const float l2 = __fmul_rn(__fsub_rn(h.hi[k], ok), ik);
        const float mx = sse_max(sse_min(l1, INFINITY), sse_min(l2, INFINITY));
        const float mn = sse_min(sse_max(l1, -INFINITY), sse_max(l2, -INFINITY));
        lmax = k == 0 ? mx : sse_min(lmax, mx);
        lmin = k == 0 ? mn : sse_max(lmin, mn);
    }
    if (!(lmax >= lmin)) return;
    const float tmn = lmin < mint ? mint : lmin;
    const float tmx = lmax > maxt ? maxt : lmax;
    if (!(tmx > tmn)) return;
    float dx = __fmul_rn(h.cell[0], ix), dy = __fmul_rn(h.cell[1], iy), dz = __fmul_rn(h.cell[2], iz);
    const float ex = __fmul_rn(__fsub_rn(__fadd_rn(o.x, __fmul_rn(d.x, tmn)), h.lo[0]), h.inv_cell[0]);
    const float ey = __fmul_rn(__fsub_rn(__fadd_rn(o.y, __fmul_rn(d.y, tmn)), h.lo[1]), h.inv_cell[1]);
    const float ez = __fmul_rn(__fsub_rn(__fadd_rn(o.z, __fmul_rn(d.z, tmn)), h.lo[2]), h.inv_cell[2]);
    // Grid::posToVoxel: Utils::clamp((int)pos, 0, res - 1)
    int px = max(0, min((int)ex, h.res[0] - 1));
    int py = max(0, min((int)ey, h.res[1] - 1));
    int pz = max(0, min((int)ez, h.res[2] - 1));
    uint32_t cell = (uint32_t)px + (uint32_t)h.res[0] * ((uint32_t)py + (uint32_t)h.res[1] * (uint32_t)pz);
    int sx = 1, sy = 1, sz = 1, cx = h.res[0], cy = h.res[1], cz = h.res[2];
    if (!(d.x >= 0.f)) { sx = -1; cx = -1; dx = -dx; }
    if (!(d.y >= 0.f)) { sy = -1; cy = -1; dy = -dy; }
    if (!(d.z >= 0.f)) { sz = -1; cz = -1; dz = -dz; }
    float lx = __fmul_rn(__fmul_rn(__fsub_rn((float)(px + (sx > 0 ? 1 : 0)), ex), ix), h.cell[0]);
    float ly = __fmul_rn(__fmul_rn(__fsub_rn((float)(py + (sy > 0 ? 1 : 0)), ey), iy), h.cell[1]);
    float lz = __fmul_rn(__fmul_rn(__fsub_rn((float)(pz + (sz > 0 ? 1 : 0)), ez), iz), h.cell[2]);
    float t = tmn;
    const int steps = h.res[0] + h.res[1] + h.res[2] + 3;
    for (int it = 0; it < steps; ++it) {
        // Vector3::argMin (Structs/Vector3.hxx:473-475)
        const int ax = (lx < ly) ? ((lx < lz) ? 0 : 2) : ((ly < lz) ? 1 : 2);
        const float la = pick3(ax, lx, ly, lz);
        const float tn = __fadd_rn(t, la);
        visit(cell, t, tmx < tn ? tmx : tn);  // std::min(t + l[minAxis], _maxt)
        t = tn;
        lx = __fsub_rn(lx, la);
        ly = __fsub_rn(ly, la);
        lz = __fsub_rn(lz, la);
        if (ax == 0) {
            lx = dx;
            cell += h.shift[0] * (uint32_t)sx;
            px += sx;
            if (px == cx) return;
        } else if (ax == 1) {
            ly = dy;
            cell += h.shift[1] * (uint32_t)sy;
            py += sy;
            if (py == cy) return;
        } else {
            lz = dz;
            cell += h.shift[2] * (uint32_t)sz;
            pz += sz;
            if (pz == cz) return;
        }
        if (!(t < tmx)) return;
    }
}

// The items of one warp's walk past the first checks of the predicate, waiting for the rest of it: the
// entry in the cell lists, the cell's t range and its selection pdf.
constexpr int kGridQueue = 64;
constexpr uint32_t kNoEntry = 0xffffffffu;
struct GridQueue {
    float tmin[kGridQueue], tmax[kGridQueue], pdf[kGridQueue];
    uint32_t at[kGridQueue];
    __align__(16) float ray[3][8];  // the query's line for each axis (grid_maybe)
};

// The per-query draws of the OFFSET, RESAMPLE_FIXED and SAMPLED reductions (Grid.hxx:466-548).  The
// reference takes them from the grid's one sequential stream in the order the queries are made;
// here each is a function of (seed, query, segment, cell, draw), the same uniform distribution
// whatever the order of evaluation: a SplitMix64 finaliser, 24 bits to [0, 1).
__device__ __forceinline__ unsigned long long splitmix64(unsigned long long z)
{
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ float grid_draw(unsigned long long key, uint32_t j)
{
    return (float)(splitmix64(key + (unsigned long long)j * 0xD1B54A32D192ED03ull) >> 40) * 0x1p-24f;
}

// Whether PhotonBeam::testIntersectionBeamBeam may accept a beam within the query's t range [tmin, tmax]
// of a cell: its first two checks (the lines' distance, t1 within the range), on the beam's line with a
// direction d2 = (1, m, n) of length up to sqrt(3), without the division and with fused multiply-adds.  The
// checks are wider than the rounding of both sides; with M = mag, the sum of the coordinates' bounds, and unit
// directions (within 1e-6):
//   ad = x . (d1 x d2) / |d2| differs from the reference's by at most 2e-6 M, taken as a = 4e-6 M, the squared
//   sine by 6e-4 of it where the predicate does not reject the pair as near-parallel; ad'^2 < r^2 sin'^2 gives
//   ad^2 <= (1 + 1/16) ad'^2 + 17 a^2 < 1.07 r^2 sin^2 + c0;
//   t1 = k / s2, k = (x.d1) |d2|^2 - b (x.d2), s2 = |d1 x d2|^2: k differs by at most 1.2e-5 M and s2 by 9e-6,
//   so a t1 in the range keeps k within [tmin s2, tmax s2] widened by slack + 1.2e-5 tmax, slack = 2.5e-5 M.
// NaN and infinite bounds pass.  The whole predicate in the reference's order decides in `finish`.
// ray: the query's line for each axis, [axis] = {o_a, o_u, o_v, d_a, d_u, d_v}, o relative to the box's middle.
__device__ __forceinline__ bool grid_maybe(const float (*ray)[8], float4 line, float r2, float tmin, float tmax,
                                           float slack, float c0)
{
    const float* f = ray[min(__float_as_int(line.z) & 3, 2)];
    const float4 f0 = *reinterpret_cast<const float4*>(f);
    const float2 f1 = *reinterpret_cast<const float2*>(f + 4);
    const float m = line.z, n = line.w, da = f0.w, du = f1.x, dv = f1.y;
    const float xa = -f0.x, xu = line.x - f0.y, xv = line.y - f0.z;
    const float ca = fmaf(du, n, -(dv * m)), cu = fmaf(-da, n, dv), cv = fmaf(da, m, -du);
    const float ad = fmaf(xa, ca, fmaf(xu, cu, xv * cv)), s2 = fmaf(ca, ca, fmaf(cu, cu, cv * cv));
    const float b = fmaf(du, m, fmaf(dv, n, da)), dd = fmaf(m, m, fmaf(n, n, 1.f));
    const float xd1 = fmaf(xa, da, fmaf(xu, du, xv * dv)), xd2 = fmaf(xu, m, fmaf(xv, n, xa));
    const float k = fmaf(-b, xd2, xd1 * dd), sl = fmaf(1.2e-5f, tmax, slack);
    return !(ad * ad > fmaf(1.07f * r2, s2, c0)) && !(k < fmaf(tmin, s2, -sl)) && !(k > fmaf(tmax, s2, sl));
}

// BB1D of one query by one warp over the beam grid.  The walk runs on every lane alike.  The entries of a
// visited cell (max_beams_in_cell items of an over-full cell of a reduced grid, Grid.hxx:453-548) go 32 at a
// time, one per lane, through the first checks of PhotonBeam::testIntersectionBeamBeam (grid_maybe: the distance
// of the two lines, then the closest point's t1 within the cell's t range), on their 16-byte lines.  Whole
// batches of consecutive entries are checked at once, the next batch's lines loaded ahead; a cell's last items
// and the items of reduced cells wait in the lanes' registers until the warp is full.  What passes goes to a
// queue in shared memory, whose 32-wide batches run the rest: the medium, the whole predicate, the radius, and
// PhotonBeam::accumulate / accumulate2 (PhotonBeam.hxx:315-367, 375-480) divided by the cell's selection pdf.
//
// Bound by instruction issue and the loads' latency: at cube512 over a 64^3 grid a query checks 15,000 entries
// and takes 1,260.  With the cells queued in shared memory, two 16-byte loads per entry, the predicate's own
// checks and batches that ended with the queue 37.0 ms, now 29.8 ms (128^3: 37.3 -> 33.8, cube128 over 64^3:
// 1.06 -> 0.81, cube1024 over 64^3: 511 -> 399; mixed mode).  Cells' last entries as partly filled batches: 31.8
// instead of 29.0 ms (an earlier version of the contribution).
template <bool kMixed>
__device__ __forceinline__ Rgb bb1d_query_grid(const GatherConsts& K, const DMedium* media, const LightSoA& Lv,
                                               const BeamGrid& G, const GridHeader& hdr, const BeamSoA& Bs,
                                               const SegQueriesDev& Q, int64_t q, SegCtx& s, GridQueue& gq,
                                               int lane, unsigned long long& cnt, unsigned long long& h,
                                               unsigned long long& tested)
{
    const unsigned lt = (1u << lane) - 1u;
    unsigned cnt32 = 0, tested32 = 0;
    const Rgb res = segment_loop(K, media, Q, q, s, [&](const DMedium& m) {
        Rgb part = rgb(0.f);
        const int mid = (int)(&m - media);
        int held = 0, nq = 0;  // the lanes that hold an item, and items past the first checks (warp-uniform)
        // the lane's item: its entry, the cell's t range and selection pdf, the entry's geometry
        uint32_t at = kNoEntry;
        float imin = 0.f, imax = 0.f, ipdf = 1.f;
        float4 line = make_float4(0.f, 0.f, 0.f, 0.f);
        float r2 = G.r2;
        // the bounds of grid_maybe
        float mag = fabsf(s.o.x) + fabsf(s.o.y) + fabsf(s.o.z);
        for (int k = 0; k < 3; ++k) mag += fmaxf(fabsf(hdr.lo[k]), fabsf(hdr.hi[k]));
        if (!(fabsf(s.d.x * s.d.x + s.d.y * s.d.y + s.d.z * s.d.z - 1.f) <= 1e-6f)) mag = __int_as_float(0x7f800000);
        const float slack = 2.5e-5f * mag, c0 = 2.72e-10f * mag * mag;
        __syncwarp();
        if (lane < 3) {
            const float o[3] = {s.o.x - 0.5f * (hdr.lo[0] + hdr.hi[0]), s.o.y - 0.5f * (hdr.lo[1] + hdr.hi[1]),
                                s.o.z - 0.5f * (hdr.lo[2] + hdr.hi[2])};
            float* f = gq.ray[lane];
            f[0] = pick3(lane, o[0], o[1], o[2]);
            f[1] = pick3(lane, o[1], o[2], o[0]);
            f[2] = pick3(lane, o[2], o[0], o[1]);
            f[3] = pick3(lane, s.d.x, s.d.y, s.d.z);
            f[4] = pick3(lane, s.d.y, s.d.z, s.d.x);
            f[5] = pick3(lane, s.d.z, s.d.x, s.d.y);
        }
        __syncwarp();
        auto finish = [&](int k) {
            const uint32_t at = gq.at[k];
            const int b = __ldg(&G.ptr[at]);
            if (__ldg(&G.medium[b]) != mid) return;  // mMedium == medium
            const float4 a = __ldg(&G.beam_a[b]), bd = __ldg(&G.beam_b[b]);
            const V3 o2 = v3(a.x, a.y, a.z), d2 = v3(bd.x, bd.y, bd.z);
            float dist, sinT, t1, t2;
            if (!test_beam_beam(s.o, s.d, gq.tmin[k], gq.tmax[k], o2, d2, 0.f, a.w, bd.w, &dist, &sinT, &t1, &t2))
                return;
            const float rs = beam_start_radius(Bs, kMixed ? &G.pay[b].lv.z : &Bs.radius[b]);
            const float radius = beam_radius_at(Bs, b, rs, t2);
            if (radius < dist) return;  // PhotonBeam.hxx:334-336 / 411-413
            ++cnt32;
            h += mix64((unsigned long long)b);
            Rgb c;
            if (kMixed) {
                // the beam's packed payload, and the FP64 closest approach of near-parallel lines
                // (the candidate decision above stays FP32)
                const float cb = s.d.x * d2.x + s.d.y * d2.y + s.d.z * d2.z;
                if (1.f - cb * cb < 1e-2f) closest_approach_f64(s.o, s.d, o2, d2, dist, sinT, t1, t2);
                c = bb1d_contrib_packed<false>(K, m, s, G.pay[b], PairGeo{xdot3(s.d, d2), dist * dist, sinT, t1, t2},
                                               beam_radius_at(Bs, b, rs, t2));
            } else {
                c = bb1d_contrib<false>(K, m, Lv, Bs, s, b, o2, d2, radius, dist, sinT, t1, t2);
            }
            const float pdf = gq.pdf[k];
            if (pdf != 1.f) c = c * __fdiv_rn(1.f, pdf);
            part = part + c;
        };
        // 32 items through the first checks, those that pass into the queue; `last`: and the queue's last ones
        auto check = [&](bool valid, uint32_t entry, float4 ln, float rr, float tmin, float tmax, float pdf, bool last) {
            const bool near = valid && grid_maybe(gq.ray, ln, rr, tmin, tmax, slack, c0);
            const unsigned bal = __ballot_sync(kFull, near);
            if (near) {
                const int slot = nq + __popc(bal & lt);
                gq.tmin[slot] = tmin;
                gq.tmax[slot] = tmax;
                gq.pdf[slot] = pdf;
                gq.at[slot] = entry;
            }
            nq += __popc(bal);
            while (nq >= 32 || (last && nq > 0)) {
                const int n = min(nq, 32);
                nq -= n;
                __syncwarp();
                if (lane < n) finish(nq + lane);
                __syncwarp();
            }
        };
        // the reductions' draws of this query and segment
        const unsigned long long qkey =
            splitmix64(((unsigned long long)(uint32_t)hdr.seed << 32) ^ (unsigned long long)q) ^
            ((unsigned long long)__float_as_uint(s.dmin) * 0x94D049BB133111EBull);
        grid_walk(hdr, s.o, s.d, s.dmin, s.dmax, [&](uint32_t cell, float cmin, float cmax) {
            const uint32_t begin = __ldg(&G.cells[cell]);
            const uint32_t beams = __ldg(&G.cells[cell + 1]) - begin;
            const float pdf = G.pdf ? __ldg(&G.pdf[cell]) : 1.f;
            // a reduced cell tests max_beams beams, SAMPLED draws for each of them
            const uint32_t n = (pdf != 1.f && hdr.reduction != 3) ? hdr.max_beams : beams;
            // whole batches of an unreduced cell: 32 consecutive entries, the next ones loaded ahead
            const uint32_t whole = pdf == 1.f || hdr.reduction == 0 ? n & ~31u : 0u;
            float4 ahead = line;
            if (whole) ahead = __ldg(&G.line[begin + (uint32_t)lane]);
            for (uint32_t pos = 0; pos < n;) {
                if (pos < whole) {
                    const uint32_t entry = begin + pos + (uint32_t)lane;
                    const float4 ln = ahead;
                    pos += 32;
                    ++tested32;
                    if (pos < whole) ahead = __ldg(&G.line[entry + 32]);
                    check(true, entry, ln, G.line_r2 ? __ldg(&G.line_r2[entry]) : G.r2, cmin, cmax, pdf, false);
                    continue;
                }
                // the last items of a cell wait in the lanes until 32 are there
                const uint32_t j = pos + (uint32_t)(lane - held);
                if (lane >= held && j < n) {
                    // the entry of item j: intersectPresampled / intersectOffsetted / intersectFixedSampled /
                    // intersectSampled (Grid.hxx:453-548); unreduced cells and PRESAMPLE: the j-th of the list
                    at = begin + j;
                    if (pdf != 1.f && hdr.reduction != 0) {
                        const unsigned long long key = splitmix64(qkey + (unsigned long long)cell * 0x9E3779B97F4A7C15ull);
                        if (hdr.reduction == 1) {
                            const uint32_t off = (uint32_t)__fmul_rn(grid_draw(key, 0), (float)beams);
                            const uint32_t k = min(hdr.max_beams, beams - min(off, beams));
                            at = j < k ? begin + off + j : begin + (j - k);
                        } else if (hdr.reduction == 2) {
                            at = begin + min((uint32_t)__fmul_rn(grid_draw(key, j), (float)beams), beams - 1);
                        } else if (!(grid_draw(key, j) < pdf)) {
                            at = kNoEntry;
                        }
                    }
                    imin = cmin;
                    imax = cmax;
                    ipdf = pdf;
                    if (at != kNoEntry) {
                        ++tested32;
                        line = __ldg(&G.line[at]);
                        if (G.line_r2) r2 = __ldg(&G.line_r2[at]);
                    }
                }
                const int took = (int)min(n - pos, (uint32_t)(32 - held));
                pos += (uint32_t)took;
                held += took;
                if (held == 32) {
                    held = 0;
                    check(at != kNoEntry, at, line, r2, imin, imax, ipdf, false);
                }
            }
        });
        if (held > 0 || nq > 0) check(lane < held && at != kNoEntry, at, line, r2, imin, imax, ipdf, true);
        return part;
    });
    cnt += cnt32;
    tested += tested32;
    return res;
}

// Persistent, one warp per query from the atomic work queue.  5 blocks of 4 warps per SM, between the spills of more
// and the empty SMs of fewer: over 64^3 cells 4 / 5 / 6 blocks take 420 / 399 / 412 ms at cube1024, 726 / 681 / 698 at
// boxes3, 29.6 / 29.8 / 31.0 at cube512 and 0.76 / 0.81 / 0.84 at cube128 (mixed mode; plain mode at cube512
// 42.1 / 40.7 / 43.2).
template <bool kMixed>
__global__ void __launch_bounds__(128, 5) k_bb1d_grid(const __grid_constant__ GatherConsts K, const LightSoA Lv,
                                                  const BeamGrid G, const BeamSoA Bs, const SegQueriesDev Q,
                                                  const upbp_mis* __restrict__ cam, const CamSum* __restrict__ cs,
                                                  const Outputs O, unsigned int* __restrict__ work,
                                                  const int32_t* __restrict__ order)
{
    constexpr int kWarps = 4;
    __shared__ DMedium media[UPBP_MAX_MEDIA];
    __shared__ GridHeader s_hdr;
    __shared__ GridQueue s_q[kWarps];
    __shared__ upbp_mis s_e[kWarps];
    __shared__ CamSum s_cs[kWarps];
    if (threadIdx.x == 0) s_hdr = *G.hdr;
    stage_media(K, media);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (;;) {
        unsigned qq = 0;
        if (lane == 0) qq = atomicAdd(work, 1u);
        const int64_t item = (int64_t)__shfl_sync(kFull, qq, 0);
        if (item >= Q.n) break;
        const int64_t q = order ? (int64_t)__ldg(&order[item]) : item;
        Rgb acc = rgb(0.f);
        unsigned long long cnt = 0, h = 0, tested = 0;
        if ((Q.flags[q] & UPBP_Q_BB1D) && (K.P.techniques & UPBP_BB1D)) {
            SegCtx s;
            init_seg_ctx<kMixed>(s, K, Q, cam, cs, q, &s_e[warp], &s_cs[warp], lane == 0);
            __syncwarp();
            acc = bb1d_query_grid<kMixed>(K, media, Lv, G, s_hdr, Bs, Q, q, s, s_q[warp], lane, cnt, h, tested);
        }
        const float r = warp_sum(acc.r), g = warp_sum(acc.g), b = warp_sum(acc.b);
        cnt = warp_sum_u64(cnt);
        h = warp_sum_u64(h);
        tested = warp_sum_u64(tested);
        if (lane == 0) {
            if (O.tested && tested) atomicAdd(O.tested, tested);
            O.rgb[3 * q + 0] = r;
            O.rgb[3 * q + 1] = g;
            O.rgb[3 * q + 2] = b;
            if (O.count) O.count[q] = (uint32_t)cnt;
            if (O.hash) O.hash[q] = h;
            const Rgb thr{Q.throughput[3 * q], Q.throughput[3 * q + 1], Q.throughput[3 * q + 2]};
            splat(O.image, Q.pixel[q], thr * K.P.norm_bb1d * Rgb{r, g, b});
        }
    }
}

}  // namespace

int bb1d_grid_blocks_per_sm(bool mixed)
{
    int nb = 0;
    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_bb1d_grid<true>, 128, 0);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_bb1d_grid<false>, 128, 0);
    return nb > 0 ? nb : 1;
}

void launch_bb1d_grid(const GatherConsts& K, const LightSoA& L, const BeamGrid& G, const BeamSoA& S,
                      const SegQueriesDev& Q, const upbp_mis* cam, const CamSum* cs, const Outputs& O, int grid,
                      bool mixed, unsigned int* work, const int32_t* order, cudaStream_t stream)
{
    if (Q.n <= 0) return;
    if (mixed) k_bb1d_grid<true><<<grid, 128, 0, stream>>>(K, L, G, S, Q, cam, cs, O, work, order);
    else k_bb1d_grid<false><<<grid, 128, 0, stream>>>(K, L, G, S, Q, cam, cs, O, work, order);
}

void launch_gather_bp2d(const GatherConsts& K, const BeamBVH& B, const BeamSoA& S, const PointQueriesDev& Q,
                        const Outputs& O, int block, cudaStream_t stream)
{
    if (Q.n <= 0) return;
    const int grid = (int)((Q.n + block - 1) / block);
    k_gather_bp2d<<<grid, block, 0, stream>>>(K, B, S, Q, O);
}

int bp2d_warp_blocks_per_sm()
{
    int nb = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_bp2d_warp<4, 6>, 128, 0);
    return nb > 0 ? nb : 1;
}

void launch_bp2d_warp(const GatherConsts& K, const BeamBVH& B, const BeamSoA& S, const PointQueriesDev& Q,
                      const Outputs& O, int grid, unsigned int* work, int* status, cudaStream_t stream)
{
    if (Q.n > 0) k_bp2d_warp<4, 6><<<grid, 128, 0, stream>>>(K, B, S, Q, O, work, status);
}

void launch_gather_pb2d(const GatherConsts& K, const LightSoA& L, const PhotonBVH& B, const SegQueriesDev& Q,
                        const upbp_mis* cam, const CamSum* cs, const Outputs& O, int block, bool mixed,
                        cudaStream_t stream, const int32_t* order)
{
    if (Q.n <= 0) return;
    const int grid = (int)((Q.n + block - 1) / block);
    if (mixed) k_gather_pb2d<true><<<grid, block, 0, stream>>>(K, L, B, Q, cam, cs, O, order);
    else k_gather_pb2d<false><<<grid, block, 0, stream>>>(K, L, B, Q, cam, cs, O, order);
}

void launch_gather_bb1d(const GatherConsts& K, const LightSoA& L, const BeamBVH& B, const BeamSoA& S,
                        const SegQueriesDev& Q, const upbp_mis* cam, const CamSum* cs, const Outputs& O, int block,
                        bool mixed, cudaStream_t stream)
{
    if (Q.n <= 0) return;
    const int grid = (int)((Q.n + block - 1) / block);
    if (mixed) k_gather_bb1d<true><<<grid, block, 0, stream>>>(K, L, B, S, Q, cam, cs, O);
    else k_gather_bb1d<false><<<grid, block, 0, stream>>>(K, L, B, S, Q, cam, cs, O);
}

// The fused segment kernel at 5 (variant 3) or 6 (variant 4) blocks of 4 warps per SM.
int segments_warp_blocks_per_sm(bool mixed, int variant)
{
    int nb = 0;
    const bool six = variant == 4;
    if (mixed) {
        if (six) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_segments_warp<true, 4, 6>, 128, 0);
        else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_segments_warp<true, 4, 5>, 128, 0);
    } else {
        if (six) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_segments_warp<false, 4, 6>, 128, 0);
        else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_segments_warp<false, 4, 5>, 128, 0);
    }
    return nb > 0 ? nb : 1;
}

void launch_segments_warp(const GatherConsts& K, const LightSoA& L, const PhotonBVH& P, const BeamBVH& B,
                          const BeamSoA& S, const SegQueriesDev& Q, const upbp_mis* cam, const CamSum* cs,
                          const Outputs& Opb, const Outputs& Obb, int grid, bool mixed, unsigned int* work,
                          int* status, const int32_t* order, cudaStream_t stream, int variant)
{
    if (Q.n <= 0) return;
    const bool six = variant == 4;
#define UPBP_SEG_LAUNCH(M, N) \
    k_segments_warp<M, 4, N><<<grid, 128, 0, stream>>>(K, L, P, B, S, Q, cam, cs, Opb, Obb, work, status, order)
    if (mixed) {
        if (six) UPBP_SEG_LAUNCH(true, 6);
        else UPBP_SEG_LAUNCH(true, 5);
    } else {
        if (six) UPBP_SEG_LAUNCH(false, 6);
        else UPBP_SEG_LAUNCH(false, 5);
    }
#undef UPBP_SEG_LAUNCH
}

// Two instantiations of the warp kernel differ only in the occupancy the compiler is asked to
// reach: 5 blocks of 4 warps per SM (up to 96 registers) or 6 (up to 80 registers, more warps to
// hide load latency, some spills); the tuning's bb1d_kernel picks 1 or 2.
template <bool kMixed>
static int blocks_for(int variant)
{
    int nb = 0;
    if (variant == 2) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_bb1d_warp<kMixed, 4, 7>, 128, 0);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_bb1d_warp<kMixed, 4, 6>, 128, 0);
    return nb > 0 ? nb : 1;
}

int pb2d_warp_blocks_per_sm(bool mixed)
{
    int nb = 0;
    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_pb2d_warp<true, 4, 6>, 128, 0);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_pb2d_warp<false, 4, 6>, 128, 0);
    return nb > 0 ? nb : 1;
}

void launch_pb2d_warp(const GatherConsts& K, const LightSoA& L, const PhotonBVH& P, const SegQueriesDev& Q,
                      const upbp_mis* cam, const CamSum* cs, const Outputs& O, int grid, bool mixed,
                      unsigned int* work, int* status, const int32_t* order, cudaStream_t stream)
{
    if (Q.n <= 0) return;
    if (mixed) k_pb2d_warp<true, 4, 6><<<grid, 128, 0, stream>>>(K, L, P, Q, cam, cs, O, work, status, order);
    else k_pb2d_warp<false, 4, 6><<<grid, 128, 0, stream>>>(K, L, P, Q, cam, cs, O, work, status, order);
}

int bb1d_warp_blocks_per_sm(bool mixed, int variant)
{
    return mixed ? blocks_for<true>(variant) : blocks_for<false>(variant);
}

// Behind the packet gather (elsewhere) this one may start as soon as all blocks of that run: its blocks take what
// the last packets leave idle.  On a second stream they did so too, but there the kernel waited for room in a
// hardware queue that another context's stream may share, and held up that one's build: two contexts
// in turn took 194.5 or 203.6 ms per step at cube1024, by the luck of the streams' queues, now 194.4.
cudaError_t launch_bb1d_warp(const GatherConsts& K, const LightSoA& L, const BeamBVH& B, const BeamSoA& S,
                             const SegQueriesDev& Q, const upbp_mis* cam, const CamSum* cs, const Outputs& O, int grid,
                             bool mixed, unsigned int* work, int* status, const int32_t* order, cudaStream_t stream,
                             int variant, const unsigned* elsewhere)
{
    if (Q.n <= 0) return cudaSuccess;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(128);
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = elsewhere ? 1 : 0;
    auto* f = variant == 2 ? (mixed ? k_bb1d_warp<true, 4, 7> : k_bb1d_warp<false, 4, 7>)
                           : (mixed ? k_bb1d_warp<true, 4, 6> : k_bb1d_warp<false, 4, 6>);
    return cudaLaunchKernelEx(&cfg, f, K, L, B, S, Q, cam, cs, O, work, status, order, elsewhere);
}

namespace {
// The contributions' inputs of every beam; the emission of the pieces copies them into its order.
__global__ void k_beam_payload(int n, const float4* __restrict__ bm_thr, const float4* __restrict__ bm_pdf,
                               const int2* __restrict__ bm_link, const float* __restrict__ bm_radius,
                               const int4* __restrict__ lv_info, const upbp_mis* __restrict__ lv_mis,
                               const LightSum* __restrict__ sums, PiecePayload* __restrict__ out)
{
    const int beam = blockIdx.x * blockDim.x + threadIdx.x;
    if (beam >= n) return;
    const int lv = bm_link[beam].x;
    // without MIS (lv_info == nullptr) the beams need not have light vertices
    upbp_mis m{};
    int4 info = make_int4(0, 0, 0, 0);
    LightSum ls{};
    if (lv_info) {
        m = load_mis(lv_mis + lv);
        info = lv_info[lv];
        ls = sums[lv];
    }
    const bool onDelta = (m.flags & UPBP_MIS_ON_LIGHT_SOURCE) && (m.flags & UPBP_MIS_IS_DELTA);
    const float4 thr = bm_thr[beam], pdf = bm_pdf[beam];
    const uint32_t bflags = (uint32_t)__float_as_int(thr.w), brsf = (uint32_t)__float_as_int(pdf.w);
    PiecePayload p;
    p.thr = make_float4(thr.x, thr.y, thr.z, (float)ls.d);
    p.pdf = make_float4(pdf.x, pdf.y, pdf.z, (float)ls.e);
    const unsigned bits = (unsigned)(info.y & kPayPathMask) | ((info.z & UPBP_LV_IS_FINITE) ? (unsigned)kPayFinite : 0u) |
                          ((bflags & UPBP_SHORT_BEAM) ? (unsigned)kPayShortBeam : 0u) |
                          ((brsf & UPBP_ORIGIN_IN_MEDIUM) ? kPayOriginInMedium : 0u);
    p.lv = make_float4(onDelta ? 0.f : fabsf(m.cos_theta_out), ls.bptb, bm_radius[beam], __int_as_float((int)bits));
    out[beam] = p;
}

// Morton code of the middle of a segment query's span (10 bits per axis in the given box).
// Spreads the low 10 bits of v to every third bit (3-D Morton interleave).
__device__ __forceinline__ uint32_t spread3(uint32_t v)
{
    uint32_t r = 0;
    for (int b = 0; b < 10; ++b) r |= ((v >> b) & 1u) << (3 * b);
    return r;
}
// Spreads the low 14 bits of v to every second bit (2-D Morton interleave).
__device__ __forceinline__ uint32_t spread2(uint32_t v)
{
    uint32_t r = 0;
    for (int b = 0; b < 14; ++b) r |= ((v >> b) & 1u) << (2 * b);
    return r;
}

// Sort key of a segment query (30 bits), by `mode` (upbp_tuning.query_order):
//  0: 3-D Morton code of the midpoint of the query's span;
//  1: camera rays (path length 1) first, along a 2-D Morton curve of their pixels (neighbouring
//     pixels' rays cross nearly the same beam pieces), then the other segments by midpoint;
//  2: 5-D Morton code of the midpoint (6 bits per axis) and the direction (octahedral map, 6 bits
//     per axis).
__global__ void k_query_keys(const SegQueriesDev Q, const float* __restrict__ bb, int mode, int width, uint32_t* keys,
                             int32_t* iota)
{
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (q >= Q.n) return;
    const int sb = Q.seg_begin[q], sc = Q.seg_count[q];
    const float t = sc > 0 ? 0.5f * (Q.seg_dist_min[sb] + Q.seg_dist_max[sb + sc - 1]) : 0.f;
    const float tm = isfinite(t) ? t : (sc > 0 ? Q.seg_dist_min[sb] : 0.f);
    float p[3];
    for (int c = 0; c < 3; ++c) p[c] = Q.origin[3 * q + c] + Q.direction[3 * q + c] * tm;
    uint32_t ix[3];
    for (int c = 0; c < 3; ++c) {
        const float ext = bb[3 + c] - bb[c];
        const float u = ext > 0.f ? (p[c] - bb[c]) / ext : 0.f;
        ix[c] = (uint32_t)fminf(fmaxf(u * 1024.f, 0.f), 1023.f);
    }
    uint32_t code = (spread3(ix[0]) << 2) | (spread3(ix[1]) << 1) | spread3(ix[2]);
    if (mode == 1) {
        const int px = Q.pixel[q];
        if (Q.path_length[q] == 1 && px >= 0 && width > 0)
            code = spread2((uint32_t)(px % width) & 0x3fffu) | (spread2((uint32_t)(px / width) & 0x3fffu) << 1);
        else
            code = (1u << 29) | (code >> 1);
    } else if (mode == 2) {
        // octahedral map of the direction to [0, 1)^2
        const float dx = Q.direction[3 * q], dy = Q.direction[3 * q + 1], dz = Q.direction[3 * q + 2];
        const float n = fabsf(dx) + fabsf(dy) + fabsf(dz);
        float ox = n > 0.f ? dx / n : 0.f, oy = n > 0.f ? dy / n : 0.f;
        if (dz < 0.f) {
            const float tx = (1.f - fabsf(oy)) * (ox >= 0.f ? 1.f : -1.f);
            oy = (1.f - fabsf(ox)) * (oy >= 0.f ? 1.f : -1.f);
            ox = tx;
        }
        const uint32_t a[5] = {ix[0] >> 4, ix[1] >> 4, ix[2] >> 4,
                               (uint32_t)fminf(fmaxf((ox * 0.5f + 0.5f) * 64.f, 0.f), 63.f),
                               (uint32_t)fminf(fmaxf((oy * 0.5f + 0.5f) * 64.f, 0.f), 63.f)};
        code = 0;
        for (int b = 5; b >= 0; --b)
            for (int k = 0; k < 5; ++k) code = (code << 1) | ((a[k] >> b) & 1u);
    }
    keys[q] = code;
    iota[q] = (int32_t)q;
}
// Sum of the per-query PB2D candidate counts (integer, so the order of the atomics does not matter).
__global__ void k_sum_counts(const uint32_t* __restrict__ cnt, int64_t n, unsigned long long* sum)
{
    unsigned long long v = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        v += cnt[i];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(sum, v);
}

// BB1D work order: the queries whose PB2D candidate count exceeds `factor` times the mean come
// first (they are the heaviest BB1D queries too), each group in Morton order of the midpoints.
// Without counts (cnt NULL) none is heavy.  The queries that packets hold (in_packet, or NULL; none where
// *held is 0) go last.
__global__ void k_heavy_keys(const uint32_t* __restrict__ cnt, int64_t n, const unsigned long long* __restrict__ sum,
                             unsigned factor, const uint32_t* __restrict__ morton,
                             const uint8_t* __restrict__ in_packet, const unsigned* __restrict__ held, uint32_t* keys,
                             int32_t* iota)
{
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (q >= n) return;
    const bool heavy = cnt && (unsigned long long)cnt[q] * (unsigned long long)n > (unsigned long long)factor * *sum;
    keys[q] = in_packet && in_packet[q] && *held ? 0xffffffffu : (heavy ? 0u : (1u << 30)) | morton[q];
    iota[q] = (int32_t)q;
}
}  // namespace

void launch_heavy_keys(const uint32_t* cnt, int64_t n, unsigned long long* sum, unsigned factor,
                       const uint32_t* morton, const uint8_t* in_packet, const unsigned* held, uint32_t* keys,
                       int32_t* iota, cudaStream_t stream)
{
    if (n <= 0) return;
    if (cnt) k_sum_counts<<<148 * 4, 256, 0, stream>>>(cnt, n, sum);
    k_heavy_keys<<<(int)((n + 255) / 256), 256, 0, stream>>>(cnt, n, sum, factor, morton, in_packet, held, keys, iota);
}

void launch_beam_payload(int n, const float4* bm_thr, const float4* bm_pdf, const int2* bm_link, const float* bm_radius,
                         const int4* lv_info, const upbp_mis* lv_mis, const LightSum* sums, PiecePayload* out,
                         cudaStream_t stream)
{
    if (n > 0)
        k_beam_payload<<<(n + 255) / 256, 256, 0, stream>>>(n, bm_thr, bm_pdf, bm_link, bm_radius, lv_info, lv_mis, sums,
                                                            out);
}

void launch_query_keys(const SegQueriesDev& Q, const float* bbox, int mode, int image_width, uint32_t* keys,
                       int32_t* iota, cudaStream_t stream)
{
    if (Q.n > 0) k_query_keys<<<(int)((Q.n + 255) / 256), 256, 0, stream>>>(Q, bbox, mode, image_width, keys, iota);
}

void launch_gather_pp3d(const GatherConsts& K, const LightSoA& L, const HashGridDev& G, const PointQueriesDev& Q,
                        const upbp_mis* cam, const CamSum* cs, const Outputs& O, int block, bool mixed,
                        cudaStream_t stream)
{
    if (Q.n <= 0) return;
    const int grid = (int)((Q.n * 8 + block - 1) / block);
    if (mixed) k_gather_pp3d<true><<<grid, block, 0, stream>>>(K, L, G, Q, cam, cs, O);
    else k_gather_pp3d<false><<<grid, block, 0, stream>>>(K, L, G, Q, cam, cs, O);
}

}  // namespace upbp
