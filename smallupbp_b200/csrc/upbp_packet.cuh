// Packets of camera rays for BB1D (upbp_packet.cu).
#pragma once

#include "upbp_kernels.cuh"

namespace upbp {

constexpr int kPacketParts = 8;  // work items of a packet at most

struct PacketTotals {
    unsigned long long weight;
    unsigned queries;  // queries in packets
    unsigned items;
};

// The 8 x 4 pixel blocks of the image and their queries in the pixel order.
struct PacketsDev {
    int2* range;                  // per block: its first query in the order, and how many
    uint32_t* weight;             // per block: work estimate, 0 where the block is no packet
    uint32_t* key;                // per item slot (kPacketParts per block): weight, 0 for none
    uint32_t* item;               // block | part << 24 | log2(parts) << 28
    const uint32_t* item_sorted;  // heaviest first
    uint8_t* in_packet;           // per query: whether a packet holds it (zeroed by the caller)
    PacketTotals* totals;         // zeroed by the caller
};

int packet_blocks(int width, int height);
// resident: blocks of the gather that run at a time
void launch_packet_setup(const SegQueriesDev& Q, const uint32_t* keys, const int32_t* order, const uint32_t* cnt_pb2d,
                         int width, int height, const float* bbox, float piece_len, int resident, const PacketsDev& P,
                         cudaStream_t s);
int bb1d_packet_blocks_per_sm(bool mixed);
void launch_bb1d_packet(const GatherConsts& K, const LightSoA& L, const BeamBVH& B, const BeamSoA& S,
                        const SegQueriesDev& Q, const Outputs& O, const int32_t* order, const PacketsDev& P,
                        const float* bbox, float piece_len, int grid, bool mixed, unsigned* work, cudaStream_t s);

}  // namespace upbp
