// Packets of camera rays for BB1D (upbp_packet.cu).
#pragma once

#include "upbp_kernels.cuh"

namespace upbp {

constexpr int kPacketParts = 8;  // work items of a packet at most

// Packets are made of this many camera queries (path length 1, on a pixel) and more: fewer do not keep the blocks
// busy to the end.  Against one warp per query BB1D takes, with packets (cube scenes with LONG, SHORT and few beams,
// nested boxes, KNN radii; mixed / plain mode): at 51 thousand camera queries 0.79-1.14 / 0.78-1.20 of the time,
// at 66 thousand 0.75-1.10 / 0.74-1.21, at 84 thousand 0.68-0.96 / 0.69-1.03, at 114 thousand 0.65-0.87 /
// 0.67-0.97, at 200 thousand and more 0.6-0.8.
constexpr unsigned kPacketCamera = 80000;

struct PacketTotals {
    unsigned long long weight;
    unsigned camera;  // queries in the pixel order
    unsigned rays;    // those that a packet could hold
    unsigned packets;
    unsigned items;
    unsigned queries;  // queries in packets: rays, or 0 where the camera queries are too few
};

// The packets among the 8 x 4 pixel blocks of the queries, and the work items made of them.
struct PacketsDev {
    int2* range;        // per packet: its first query in the pixel order; how many, and the axis << 8
    uint32_t* weight;   // per packet: work estimate
    uint32_t* key;      // per item slot: weight (zeroed by the caller)
    unsigned long long* item;               // per item slot: a run of a packet's rays
    const unsigned long long* item_sorted;  // heaviest first
    uint8_t* in_packet;                     // per query: whether a packet could hold it (zeroed by the caller)
    PacketTotals* totals;                   // zeroed by the caller
};

// The most packets that n queries of an image can make, and the item slots for them.
int packet_max(int width, int height, int64_t n);
int packet_slots(int packets, int resident);
// packets: packet_max; resident: blocks of the gather that run at a time
void launch_packet_setup(const SegQueriesDev& Q, const uint32_t* keys, const int32_t* order, const uint32_t* cnt_pb2d,
                         int packets, int64_t n_pixels, const float* bbox, float piece_len, int resident,
                         const PacketsDev& P, cudaStream_t s);
int bb1d_packet_blocks_per_sm(bool mixed);
void launch_bb1d_packet(const GatherConsts& K, const LightSoA& L, const BeamBVH& B, const BeamSoA& S,
                        const SegQueriesDev& Q, const Outputs& O, const int32_t* order, const PacketsDev& P,
                        const float* bbox, float piece_len, int grid, bool mixed, unsigned* work, cudaStream_t s);

}  // namespace upbp
