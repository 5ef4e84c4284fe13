// Contributions of the estimators, shared by the gather kernels (upbp_gather.cu, upbp_packet.cu).
//
//  * PB2D  : breIntersectFuncHomogeneous2 (Bre/Bre.cxx:293-464)
//  * BB1D  : PhotonBeam::accumulate2 (Beams/PhotonBeam.hxx:386-607)
// and the per-segment driver of evalBre / evalBeamBeamEstimate.  Both files are compiled with the
// approximate FP32 division; the candidate predicates use explicit IEEE intrinsics.
#pragma once

#include <cfloat>
#include <cstdint>

#include "upbp_kernels.cuh"
#include "upbp_mis_prep.cuh"
#include "upbp_traverse.cuh"

namespace upbp {

namespace {

// Camera MisData as the reference array holds it during an estimator call at path length L:
// entries < L-1 from the snapshot, entry L-1 from the snapshot with mRaySampleRevPdfInv set by
// the estimator, entry L written by the estimator for the candidate.
struct CamView {
    const upbp_mis* snap;
    int L;
    const upbp_mis* cand;
    float prev_ray_rev_inv;
    __device__ upbp_mis operator()(int k) const
    {
        if (k == L) return *cand;
        upbp_mis m = load_mis(snap + k);
        if (k == L - 1) m.ray_sample_rev_pdf_inv = prev_ray_rev_inv;
        return m;
    }
};

struct CamSnap {
    const upbp_mis* snap;
    __device__ upbp_mis operator()(int k) const { return load_mis(snap + k); }
};

struct LightView {
    const upbp_mis* mis;
    int override_idx;
    float override_ray_rev_inv;
    __device__ upbp_mis operator()(int k) const
    {
        upbp_mis m = load_mis(mis + k);
        if (k == override_idx) m.ray_sample_rev_pdf_inv = override_ray_rev_inv;
        return m;
    }
};

// Per-segment state that evalBre / evalBeamBeamEstimate hand to the callbacks through
// AdditionalRayDataForMis (Bre.cxx:839-850, PhBeams.cxx:198-210).
struct SegCtx {
    V3 o, d;
    float dmin, dmax;
    float rs_pdf, rs_rev_pdf;  // mRaySamplePdf / mRaySampleRevPdf accumulated over earlier segments
    uint32_t rsf;              // mRaySamplingFlags
    int L;
    float last_pdf_w_inv;
    uint32_t ray_flags;        // beamType | estimatorTechniques
    const upbp_mis* cam;
    // mixed mode: camera entry L-1 and the FP64 suffix of the camera walk (the warp kernel keeps
    // them in shared memory: they are the same for the whole warp)
    const upbp_mis* e;
    const CamSum* cs;
};

__device__ __forceinline__ void fill_cand(upbp_mis& c, const upbp_params& P, float pdf_a_inv, float rsp_inv,
                                          float ratio, float sel_pdf, uint32_t flags)
{
    c.pdf_a_inv = pdf_a_inv;
    c.rev_pdf_a = 1.f;
    c.rev_pdf_a_without_bsdf = 1.f;
    c.ray_sample_pdf_inv = rsp_inv;
    c.ray_sample_rev_pdf_inv = 1.f;
    c.ray_sample_pdfs_ratio = ratio;
    c.ray_sample_rev_pdfs_ratio = 0.f;
    c.sin_theta = 0.f;
    c.cos_theta_out = 0.f;
    c.surf_factor = 0.f;
    c.pp3d_factor = P.mis_factor_pp3d;
    c.pb2d_factor = P.mis_factor_pb2d;
    c.bb1d_factor = P.mis_factor_bb1d;
    c.bb1d_beam_selection_pdf = sel_pdf;
    c.flags = flags;
}

// ----------------------------------------------------------------- estimators without MIS
// breIntersectFuncHomogeneous (Bre.cxx:239-291), the callback of VolLightTracer's pure PB2D: the
// photon's flux (its light vertex's throughput) x transmittance to the photon (over the
// free-flight pdf for SHORT query beams) x sigma_s x HG x the 2-D Epanechnikov kernel, with no
// rejects and no MIS weight.  The reference's expression divides the product by r^2 pi / 2.
__device__ __forceinline__ Rgb pb2d_contrib_nomis(const DMedium& m, const LightSoA& Lv, const SegCtx& s, int lv,
                                                  float t, float d2, float r2)
{
    Rgb att = eval_att(m, t - s.dmin);
    if (s.ray_flags & UPBP_SHORT_BEAM) att = att / comp(att, m.min_idx);
    const float4 ld = __ldg(&Lv.dir[lv]);
    const float4 th = __ldg(&Lv.thr[lv]);
    float sinT;
    const float phase = hg_pdf(s.d, neg3(v3(ld.x, ld.y, ld.z)), m.g, &sinT);
    const Rgb ss{m.ss[0], m.ss[1], m.ss[2]};
    return (Rgb{th.x, th.y, th.z} * att * ss * phase * (1.f - d2 / r2)) / (r2 * UPBP_PI_F * 0.5f);
}

// PhotonBeam::accumulate without MIS data (PhotonBeam.hxx:315-367), VolLightTracer's pure BB1D:
// (1 / beam selection pdf, 1 without beam reduction) x the beam's throughput x sigma_s x the query
// and beam transmittances (each over its free-flight pdf for SHORT beams) x HG x the 1-D kernel.
// The candidate test and the radius test are the caller's, as for accumulate2.
__device__ __forceinline__ Rgb bb1d_contrib_nomis(const DMedium& m, const SegCtx& s, float4 bthr, bool beam_short,
                                                  V3 bdir, float radius, float dist, float sinTheta, float t1,
                                                  float t2)
{
    Rgb att = eval_att(m, t1 - s.dmin);
    const Rgb batt = eval_att(m, t2);
    if (s.ray_flags & UPBP_SHORT_BEAM) att = att / comp(att, m.min_idx);
    att = att * batt;
    if (beam_short) att = att / comp(batt, m.min_idx);
    float sinDummy;
    const float phase = hg_pdf(s.d, bdir, m.g, &sinDummy);
    const Rgb ss{m.ss[0], m.ss[1], m.ss[2]};
    return ((1.0f * Rgb{bthr.x, bthr.y, bthr.z} * ss * att * phase * (1.f - dist * dist / (radius * radius))) * 3.f) /
           (4.f * radius * sinTheta);
}

// ----------------------------------------------------------------- PB2D contribution
// breIntersectFuncHomogeneous2 after testIntersectionBre accepted photon `lv` at (t, d2).
template <bool kMixed>
__device__ Rgb pb2d_contrib(const GatherConsts& K, const DMedium& m, const LightSoA& Lv, const SegCtx& s, int lv,
                            float t, float d2, float r2)
{
    const upbp_params& P = K.P;
    if (P.techniques & UPBP_NO_MIS) return pb2d_contrib_nomis(m, Lv, s, lv, t, d2, r2);
    const int4 info = __ldg(&Lv.info[lv]);
    const int pl = info.y;
    if ((uint32_t)(pl + s.L) > P.max_path_length || (uint32_t)(pl + s.L) < P.min_path_length) return rgb(0.f);
    if (s.L == 1 && t < P.min_dist_to_med) return rgb(0.f);
    Rgb att = eval_att(m, t - s.dmin);
    const float pdf = comp(att, m.min_idx);
    if (s.ray_flags & UPBP_SHORT_BEAM) att = att / pdf;
    float rsp = m.min_st * pdf;
    float rsr = (s.rsf & UPBP_ORIGIN_IN_MEDIUM) ? rsp : pdf;
    const float ratio = 1.0f / m.min_st;
    if (!rgb_positive(att)) return rgb(0.f);
    rsp *= s.rs_pdf;
    rsr *= s.rs_rev_pdf;
    const float4 ld = __ldg(&Lv.dir[lv]);
    float sinT;
    const float phase = hg_pdf(neg3(s.d), v3(ld.x, ld.y, ld.z), m.g, &sinT);
    if (phase <= 0.f) return rgb(0.f);
    const float camDirPdfW = phase * m.cont;
    const float camRevPdfW = phase * __ldg(&Lv.pos[lv]).w;
    const float kernel = (1.f - d2 / r2) / (r2 * UPBP_PI_F * 0.5f);  // the photon's radiusSqr
    if (!is_pos(kernel)) return rgb(0.f);
    const float4 th = __ldg(&Lv.thr[lv]);
    const Rgb ss{m.ss[0], m.ss[1], m.ss[2]};
    const Rgb unweighted = Rgb{th.x, th.y, th.z} * att * ss * phase * kernel;
    if (rgb_black_or_neg(unweighted)) return rgb(0.f);
    const float distSq = t * t;
    const float rspInv = 1.0f / rsp;
    upbp_mis cand;
    fill_cand(cand, P, s.last_pdf_w_inv * distSq * rspInv, rspInv, ratio, K.has_bb1d_beams ? 1.f : 0.f,
              (m.mfp > P.bb1d_min_mfp) ? UPBP_MIS_IN_MEDIUM_WITH_BEAMS : 0u);
    const float last = (s.ray_flags & UPBP_SHORT_BEAM) ? (float)(1.0 / (double)(ratio * cand.pb2d_factor))
                                                       : rsp / cand.pb2d_factor;
    const upbp_mis lvm = load_mis(Lv.mis + lv);
    if (kMixed) {
        const float wc = camera_weight_fast(s.L, cand, last, sinT, lvm.ray_sample_pdf_inv, lvm.ray_sample_pdfs_ratio,
                                            camRevPdfW * rsr / distSq, *s.e, 1.0f / rsr, *s.cs, s.ray_flags,
                                            P.query_beam_type, P.photon_beam_type);
        const LightSum ls = Lv.sums[lv];
        const float wl = last * ((float)ls.a + camDirPdfW * (float)ls.c);
        return (1.0f / (wl + wc)) * unweighted;
    }
    const CamView cam{s.cam, s.L, &cand, 1.0f / rsr};
    const float wCamera = camera_path_weight(s.L, last, sinT, lvm.ray_sample_pdf_inv, lvm.ray_sample_pdfs_ratio,
                                             camRevPdfW * rsr / distSq, P.query_beam_type, P.photon_beam_type,
                                             s.ray_flags, cam);
    const LightView lview{Lv.mis, -1, 0.f};
    const float wLight = light_path_weight(info.x, pl, last, 0.f, 0.f, 0.f, camDirPdfW, UPBP_PB2D, P.query_beam_type,
                                           P.photon_beam_type, s.ray_flags, Lv.path_ends, lview, nullptr);
    const float w = 1.f / (wLight + wCamera);
    return w * unweighted;
}

// ----------------------------------------------------------------- BB1D contribution
// PhotonBeam::accumulate2 after testIntersectionBeamBeam and the radius test accepted `beam`.
// FP64 closest approach of the query line and the beam line (unit directions), used in mixed
// mode for near-parallel pairs where the FP32 solve of PhotonBeam.hxx:253-293 cancels.
__device__ __forceinline__ void closest_approach_f64(V3 O1, V3 d1, V3 O2, V3 d2, float& dist, float& sinT, float& t1,
                                                     float& t2)
{
    const double ax = d1.x, ay = d1.y, az = d1.z, bx = d2.x, by = d2.y, bz = d2.z;
    const double wx = (double)O1.x - O2.x, wy = (double)O1.y - O2.y, wz = (double)O1.z - O2.z;
    const double cx = ay * bz - az * by, cy = az * bx - ax * bz, cz = ax * by - ay * bx;
    const double s2 = cx * cx + cy * cy + cz * cz;
    const double b = ax * bx + ay * by + az * bz;
    const double dd = ax * wx + ay * wy + az * wz;
    const double ee = bx * wx + by * wy + bz * wz;
    const double aa = ax * ax + ay * ay + az * az, cc = bx * bx + by * by + bz * bz;
    const double den = aa * cc - b * b;
    const double s = sqrt(s2);
    t1 = (float)((b * ee - cc * dd) / den);
    t2 = (float)((aa * ee - b * dd) / den);
    dist = (float)(fabs(-wx * cx - wy * cy - wz * cz) / s);
    sinT = (float)s;
}

// Radius of a beam at t in the reference's operations (PhotonBeam.hxx:411); rc = 0: constant.
__device__ __forceinline__ float radius_at(float rs, float rc, float t)
{
    return rc == 0.f ? rs : __fadd_rn(rs, __fmul_rn(t, rc));
}

// How far beyond its piece's interval the lines' closest point may lie, times sin(theta): 0 for an inner
// piece; the first and the last piece also own the pairs whose closest point is clamped to the beam's end,
// which the query's line then passes within the reach (the largest radius plus the margin).
__device__ __forceinline__ float piece_slack(float len, float r2max, float t_lo, float t_hi, float extra)
{
    return t_lo > 0.f && t_hi < len ? 0.f : (r2max * fast_rsqrt(r2max) + extra) * 1.01f;
}

// The decision on a pair that bb1d_pair_fast leaves open (mixed mode): the reference's FP32 predicate
// and radius test, the owner and the reach rule, in FP64 where FP32 does not decide, with the predicate's
// closest approach or, for nearly parallel lines, the FP64 one.  Returns 1 or 0.
__device__ __forceinline__ int pair_slow(V3 O1, V3 d1, float dmin, float dmax, V3 O2, V3 d2, float len, float r2max,
                                         float t_lo, float t_hi, float rs, float rc, float extra, PairGeo& g)
{
    float dist, sinT, t1, t2, b, e;
    if (!test_beam_beam(O1, d1, dmin, dmax, O2, d2, 0.f, len, r2max, &dist, &sinT, &t1, &t2, &b, &e)) return 0;
    if (radius_at(rs, rc, t2) < dist) return 0;  // PhotonBeam.hxx:411-413
    if (!piece_takes(O1, d1, dmin, dmax, O2, d2, len, t_lo, t_hi, t1, b, e, dist, rs, rc, extra)) return 0;
    if (1.f - b * b < 1e-2f) closest_approach_f64(O1, d1, O2, d2, dist, sinT, t1, t2);
    g = PairGeo{b, dist * dist, sinT, t1, t2};
    return 1;
}

template <bool kMixed>
__device__ Rgb bb1d_contrib(const GatherConsts& K, const DMedium& m, const LightSoA& Lv, const BeamSoA& Bs,
                            const SegCtx& s, int beam, V3 bo, V3 bdir, float radius, float dist, float sinTheta,
                            float t1, float t2)
{
    if (kMixed) {
        // near-parallel lines: 1 - (d1.d2)^2 small (PhotonBeam.hxx:267-273 rejects only below 1e-5)
        const float c = s.d.x * bdir.x + s.d.y * bdir.y + s.d.z * bdir.z;
        if (1.f - c * c < 1e-2f) closest_approach_f64(s.o, s.d, bo, bdir, dist, sinTheta, t1, t2);
    }
    const upbp_params& P = K.P;
    if (P.techniques & UPBP_NO_MIS) {
        const float4 bthr = __ldg(&Bs.thr[beam]);
        const bool bshort = ((uint32_t)__float_as_int(bthr.w) & UPBP_SHORT_BEAM) != 0;
        return bb1d_contrib_nomis(m, s, bthr, bshort, bdir, radius, dist, sinTheta, t1, t2);
    }
    const int2 link = __ldg(&Bs.link[beam]);
    const int lvi = link.x;
    const int4 info = __ldg(&Lv.info[lvi]);
    const int pl = info.y;
    if ((uint32_t)(pl + 1 + s.L) > P.max_path_length || (uint32_t)(pl + 1 + s.L) < P.min_path_length) return rgb(0.f);
    if (s.L == 1 && t1 < P.min_dist_to_med) return rgb(0.f);
    const float4 bthr = __ldg(&Bs.thr[beam]);
    const float4 bpdf = __ldg(&Bs.pdf[beam]);
    const uint32_t bflags = (uint32_t)__float_as_int(bthr.w);
    const uint32_t brsf = (uint32_t)__float_as_int(bpdf.w);
    // query side
    Rgb att = eval_att(m, t1 - s.dmin);
    const float pfdQ = comp(att, m.min_idx);
    if (s.ray_flags & UPBP_SHORT_BEAM) att = att / pfdQ;
    float rspQ = m.min_st * pfdQ;
    float rsrQ = (s.rsf & UPBP_ORIGIN_IN_MEDIUM) ? rspQ : pfdQ;
    const float ratioQ = 1.0f / m.min_st;
    // beam side
    const Rgb batt = eval_att(m, t2);
    att = att * batt;
    const float pfdB = comp(batt, m.min_idx);
    if (bflags & UPBP_SHORT_BEAM) att = att / pfdB;
    float rspB = m.min_st * pfdB;
    float rsrB = (brsf & UPBP_ORIGIN_IN_MEDIUM) ? rspB : pfdB;
    const float ratioB = 1.0f / m.min_st;
    if (!rgb_positive(att)) return rgb(0.f);
    rspQ *= s.rs_pdf;
    rsrQ *= s.rs_rev_pdf;
    rspB *= bpdf.x;
    rsrB *= bpdf.y;
    float sinDummy;
    const float phase = hg_pdf(neg3(s.d), neg3(bdir), m.g, &sinDummy);
    if (phase <= 0.f) return rgb(0.f);
    const float bsdfDirPdfW = phase * m.cont;
    const float bsdfRevPdfW = phase * m.cont;
    const float sel = 1.0f;  // no beam reduction (sMaxBeamsInCell == 0)
    const Rgb ss{m.ss[0], m.ss[1], m.ss[2]};
    const Rgb unweighted = ((1.0f / sel) * Rgb{bthr.x, bthr.y, bthr.z} * ss * att * phase *
                            (1.f - dist * dist / (radius * radius))) * 3.f / (4.f * radius * sinTheta);
    if (rgb_black_or_neg(unweighted)) return rgb(0.f);
    const float distSqQ = t1 * t1;
    const float rspInvQ = 1.0f / rspQ;
    upbp_mis cand;
    fill_cand(cand, P, s.last_pdf_w_inv * distSqQ * rspInvQ, rspInvQ, ratioQ, sel, UPBP_MIS_IN_MEDIUM_WITH_BEAMS);
    const bool finite = (info.z & UPBP_LV_IS_FINITE) != 0;
    const float distSqB = finite ? t2 * t2 : 1.0f;
    const float rspInvB = 1.0f / rspB;
    upbp_mis brec;
    fill_cand(brec, P, bpdf.z * distSqB * rspInvB, rspInvB, ratioB, sel, UPBP_MIS_IN_MEDIUM_WITH_BEAMS);
    float sinT = sinTheta;
    if (s.ray_flags & UPBP_NO_SINE_IN_WEIGHTS) sinT = 1.0f;
    const float f = cand.bb1d_factor;
    float last;
    if (s.ray_flags & UPBP_SHORT_BEAM)
        last = (bflags & UPBP_SHORT_BEAM) ? (float)(1.0 / (double)(ratioQ * ratioB * f * sel * sinT))
                                          : rspB / (ratioQ * f * sel * sinT);
    else
        last = (bflags & UPBP_SHORT_BEAM) ? rspQ / (ratioB * f * sel * sinT) : rspQ * rspB / (f * sel * sinT);
    const upbp_mis lvm = load_mis(Lv.mis + lvi);
    const bool onDeltaLight = (lvm.flags & UPBP_MIS_ON_LIGHT_SOURCE) && (lvm.flags & UPBP_MIS_IS_DELTA);
    const float ntl = onDeltaLight ? 0.f : bsdfDirPdfW * rsrB * fabsf(lvm.cos_theta_out) / distSqB;
    if (kMixed) {
        const float wc = camera_weight_fast(s.L, cand, last, sinT, rspInvB, ratioB, bsdfRevPdfW * rsrQ / distSqQ, *s.e,
                                            1.0f / rsrQ, *s.cs, s.ray_flags, P.query_beam_type, P.photon_beam_type);
        const LightSum ls = Lv.sums[lvi];
        float inner = ls.bptb;
        if (!(s.ray_flags & UPBP_PREVIOUS)) inner += ntl * ((float)ls.d + (float)ls.e / rsrB);
        const float wl = last * brec.pdf_a_inv * inner;
        return (1.0f / (wl + wc)) * unweighted;
    }
    const CamView cam{s.cam, s.L, &cand, 1.0f / rsrQ};
    const float wCamera = camera_path_weight(s.L, last, sinT, rspInvB, ratioB, bsdfRevPdfW * rsrQ / distSqQ,
                                             P.query_beam_type, P.photon_beam_type, s.ray_flags, cam);
    const LightView lview{Lv.mis, lvi, 1.0f / rsrB};
    const float wLight = light_path_weight(info.x, pl + 1, last, 0.f, 0.f, 0.f, ntl, UPBP_BB1D, P.query_beam_type,
                                           P.photon_beam_type, s.ray_flags, Lv.path_ends, lview, &brec);
    const float w = 1.f / (wLight + wCamera);
    return w * unweighted;
}

// PhotonBeam::accumulate2 (mixed mode) with the beam's payload packed per piece, at the lines' closest
// approach g.  kDirect: a camera path of length 1 (s.L is not read), which has no MIS records before the
// merged vertex.  The general form's operations, but for the beam's side of the weight, arranged so that neither
// the squared distance D nor the reverse pdf R along the beam is divided by:
//   wLight = last * pdfAInv * (D bptb + phase * cont * cos * (d R + e)) / rspB
// (cube1024 with the packets: 189.7 -> 187.5 ms).  With one factor for the three channels, the pdfs' products by
// reciprocals and these from the special function unit's flushing form it took 3 ms less, but pdfs below the
// normal range gave black, and the error against FP64 was up to 5 % larger.  As it is, the L2 error over six
// scenes and three seeds is 0.91 to 1.001 times the general form's.
template <bool kDirect>
__device__ __forceinline__ Rgb bb1d_contrib_packed(const GatherConsts& K, const DMedium& m, const SegCtx& s,
                                                   const PiecePayload& py, const PairGeo& g, float radius)
{
    const upbp_params& P = K.P;
    const unsigned lvbits = (unsigned)__float_as_int(py.lv.w);
    const bool bshort = (lvbits & kPayShortBeam) != 0;
    const bool qshort = (s.ray_flags & UPBP_SHORT_BEAM) != 0;
    const Rgb qatt = eval_att(m, g.t1 - s.dmin), batt = eval_att(m, g.u);
    const float pfdQ = comp(qatt, m.min_idx), pfdB = comp(batt, m.min_idx);
    Rgb att = qatt * batt;
    if (qshort) att = att / pfdQ;
    if (bshort) att = att / pfdB;
    // HG in both directions of the pair (PhaseFunction.hxx:50-80): the deflection's cosine is -d1.d2
    const float g2 = m.g * m.g, hd = 1.f + g2 + (m.g + m.g) * g.cosb;
    constexpr float inv4pi = (1.f / UPBP_PI_F) * 0.25f;
    const float phase =
        fabsf(m.g) < 1e-3f ? inv4pi : (hd > 0.f ? inv4pi * (1.f - g2) / (hd * sqrtf(hd)) : 0.f);
    const Rgb ss{m.ss[0], m.ss[1], m.ss[2]};
    const Rgb unweighted = (Rgb{py.thr.x, py.thr.y, py.thr.z} * ss * att * phase * (1.f - g.d2 / (radius * radius))) * 3.f /
                           (4.f * radius * g.sinT);
    if (P.techniques & UPBP_NO_MIS) return unweighted;
    const int L = kDirect ? 1 : s.L;
    const uint32_t length = (uint32_t)((int)(lvbits & kPayPathMask) + 1 + L);
    if (length > P.max_path_length || length < P.min_path_length || (L == 1 && g.t1 < P.min_dist_to_med) ||
        !rgb_positive(att) || phase <= 0.f || rgb_black_or_neg(unweighted))
        return rgb(0.f);
    float rspQ = m.min_st * pfdQ, rspB = m.min_st * pfdB;
    float rsrQ = (s.rsf & UPBP_ORIGIN_IN_MEDIUM) ? rspQ : pfdQ;
    float rsrB = (lvbits & kPayOriginInMedium) ? rspB : pfdB;
    rspQ *= s.rs_pdf;
    rsrQ *= s.rs_rev_pdf;
    rspB *= py.pdf.x;
    rsrB *= py.pdf.y;
    const float ratio = 1.0f / m.min_st;
    const float bsdfPdfW = phase * m.cont;
    const float rspInvQ = 1.0f / rspQ, rspInvB = 1.0f / rspB;
    const float distSqQ = g.t1 * g.t1, distSqB = (lvbits & kPayFinite) ? g.u * g.u : 1.0f;
    const bool no_sine = (s.ray_flags & UPBP_NO_SINE_IN_WEIGHTS) != 0;
    upbp_mis cand;
    fill_cand(cand, P, s.last_pdf_w_inv * distSqQ * rspInvQ, rspInvQ, ratio, 1.0f, UPBP_MIS_IN_MEDIUM_WITH_BEAMS);
    const float sinT = no_sine ? 1.0f : g.sinT;
    const float f = P.mis_factor_bb1d;
    float last;
    if (qshort) last = bshort ? (float)(1.0 / (double)(ratio * ratio * f * sinT)) : rspB / (ratio * f * sinT);
    else last = bshort ? rspQ / (ratio * f * sinT) : rspQ * rspB / (f * sinT);
    const float wc = camera_weight_fast(L, cand, last, sinT, rspInvB, ratio, bsdfPdfW * rsrQ / distSqQ, *s.e, 1.0f / rsrQ,
                                        *s.cs, s.ray_flags, P.query_beam_type, P.photon_beam_type);
    float inner = distSqB * py.lv.y;
    if (!(s.ray_flags & UPBP_PREVIOUS)) inner += bsdfPdfW * py.lv.x * (py.thr.w * rsrB + py.pdf.w);
    const float wl = last * py.pdf.z * rspInvB * inner;
    return (1.0f / (wl + wc)) * unweighted;
}

// ----------------------------------------------------------------- segment loop
// The per-segment driver of evalBre / evalBeamBeamEstimate (full and lite segments).
template <class PerSegment>
__device__ __forceinline__ Rgb segment_loop(const GatherConsts& K, const DMedium* media, const SegQueriesDev& Q,
                                            int64_t q, SegCtx& s, PerSegment&& per_segment)
{
    const uint32_t qf = Q.flags[q];
    const bool lite = (qf & UPBP_Q_LITE) != 0;
    const uint32_t qrsf = (qf & UPBP_Q_ORIGIN_IN_MEDIUM) ? UPBP_ORIGIN_IN_MEDIUM : 0u;
    const uint32_t bt = K.P.query_beam_type;
    Rgb result = rgb(0.f), attn = rgb(1.f);
    float rsp = 1.f, rsr = 1.f;
    const int sb = Q.seg_begin[q], sc = Q.seg_count[q];
    for (int i = 0; i < sc; ++i) {
        const int sg = sb + i;
        const DMedium& m = media[Q.seg_medium[sg]];
        const float dmin = Q.seg_dist_min[sg], dmax = Q.seg_dist_max[sg];
        Rgb seg = rgb(0.f);
        if (m.has_scat) {
            s.dmin = dmin;
            s.dmax = dmax;
            s.rs_pdf = rsp;
            s.rs_rev_pdf = rsr;
            s.rsf = UPBP_END_IN_MEDIUM | (i == 0 ? qrsf : 0u);
            seg = per_segment(m);
        }
        result = result + attn * seg;
        if (lite) {
            attn = attn * eval_att(m, dmax - dmin);
            float srev;
            const float spdf = ray_sample_pdf(m, dmin, dmax, i == 0 ? qrsf : 0u, &srev);
            if (!rgb_positive(attn)) break;
            rsp *= spdf;
            rsr *= srev;
        } else {
            const Rgb sa{Q.seg_attenuation[3 * sg], Q.seg_attenuation[3 * sg + 1], Q.seg_attenuation[3 * sg + 2]};
            attn = attn * (bt == UPBP_SHORT_BEAM ? sa / Q.seg_pdf[sg] : sa);
            if (!rgb_positive(attn)) break;
            rsp *= Q.seg_pdf[sg];
            rsr *= Q.seg_rev_pdf[sg];
        }
    }
    return result;
}

template <bool kMixed>
__device__ __forceinline__ void init_seg_ctx(SegCtx& s, const GatherConsts& K, const SegQueriesDev& Q,
                                             const upbp_mis* cam, const CamSum* cs, int64_t q, upbp_mis* e_store,
                                             CamSum* cs_store, bool leader = true)
{
    s.o = v3(Q.origin[3 * q], Q.origin[3 * q + 1], Q.origin[3 * q + 2]);
    s.d = v3(Q.direction[3 * q], Q.direction[3 * q + 1], Q.direction[3 * q + 2]);
    s.L = Q.path_length[q];
    s.last_pdf_w_inv = Q.last_pdf_w_inv[q];
    s.ray_flags = K.P.query_beam_type | K.P.techniques;
    s.cam = cam + Q.cam_mis_begin[q];
    s.e = e_store;
    s.cs = cs_store;
    if (kMixed && leader && !(K.P.techniques & UPBP_NO_MIS)) {
        if (s.L >= 2) *e_store = load_mis(s.cam + s.L - 1);
        *cs_store = cs[q];
    }
}

__device__ __forceinline__ void write_out(const Outputs& O, int64_t q, Rgb v, uint32_t cnt, unsigned long long h,
                                          const SegQueriesDev& Q, float norm)
{
    O.rgb[3 * q + 0] = v.r;
    O.rgb[3 * q + 1] = v.g;
    O.rgb[3 * q + 2] = v.b;
    if (O.count) O.count[q] = cnt;
    if (O.hash) O.hash[q] = h;
    const Rgb thr{Q.throughput[3 * q], Q.throughput[3 * q + 1], Q.throughput[3 * q + 2]};
    splat(O.image, Q.pixel[q], thr * norm * v);
}

}  // namespace

}  // namespace upbp
