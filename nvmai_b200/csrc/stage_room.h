// Where the decode stages' blocks find room on an SM: which register cap stage 2 takes, how an SM's memory is split, and whether
// stage 3 starts early enough to poll.  Host only, plain arithmetic.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace nvmai {

constexpr size_t kSmShared = 228 * 1024;            // an SM's shared memory; a block takes 1 KB beside its own, and 256 bytes static
constexpr size_t kBlockReserve = 1024 + 256;
constexpr uint32_t kQuarterRegs = 16384;            // registers of an SM's quarter, which holds every fourth warp of a block
constexpr uint32_t kGateUpWarps = 8, kGateUpRegs = 64, kGateUpLeanRegs = 56, kDownRegs = 56;

struct StageRoom {
    // With what most SMs hold of stage 2, one block of stage 3 fits in the shared memory: the stages ask for the whole of it
    // (launch.h).  Six layers of one row, whole / as the driver splits it: 4-bit 2048 / 512 113 / 127 us, 1024 / 1024 129 / 132, 8-bit
    // 1024 / 512 108 / 125; where it does not fit: 4-bit 2048 / 1024 with fp32 outputs 166 / 163, 8-bit 2048 / 768 182 / 177.
    bool whole_shared = false;
    // Two blocks of stage 2 an SM at most: a block of stage 3 starts beside them, and polls.
    bool early = false;
    // A block of stage 3 fits beside two of stage 2, whether or not the call's grid leaves it at two.
    bool beside_two = false;
    // Stage 2 at 56 registers: at 64 a block of stage 3 does not fit beside its blocks.  (One row, 8-bit 1024 / 512 108 us at 56, 120 at
    // 64.)  Not where that would serve a part of stage 3's blocks only (two rows of 2048 / 256, 4-bit 125 at 56, 122 at 64, 8-bit 142 /
    // 136), nor where nothing fits beside (8-bit 2048 / 768, two rows 287 / 280): there the cap only spills.
    bool lean = false;
};

// gate_up, down: shared memory of a block of stage 2 and 3; blocks, down_blocks: their grids; down_warps: warps of a block of stage 3;
// boxed: the tiles come as boxes.  (Row copies wait for stage 2 either way; there the whole memory pays from about two blocks of stage 2
// an SM on, which leave one by one: 4-bit 1024 / 576, 288 blocks, 143 us, 154 without; 2048 / 448, 224 blocks, 148, 147 without.)
inline StageRoom stage_room(size_t gate_up, size_t down, uint32_t blocks, uint32_t down_blocks, uint32_t sms, uint32_t down_warps, bool boxed) {
    StageRoom r;
    if (sms == 0) return r;
    auto fits = [&](uint32_t n) { return n * (gate_up + kBlockReserve) + down + kBlockReserve <= kSmShared; };
    r.beside_two = fits(2);
    if (!boxed) {
        r.whole_shared = 4 * blocks > 7 * sms && r.beside_two;
        return r;
    }
    // blocks an SM: the most of any up to two, above that what most SMs hold; registers allow four
    const uint32_t fullest = std::min((blocks + sms - 1) / sms, 4u), per_sm = fullest <= 2 ? fullest : std::min((blocks + sms / 2) / sms, 4u);
    r.whole_shared = fits(per_sm);
    r.early = r.whole_shared && per_sm <= 2;
    const uint32_t down_regs = (down_warps + 3) / 4 * 32 * kDownRegs;
    const uint32_t held = std::min(fullest, (uint32_t)(kSmShared / (gate_up + kBlockReserve)));      // by the shared memory
    r.lean = r.whole_shared && (held > 2 || down_blocks <= sms) && held * (kGateUpWarps / 4) * 32 * kGateUpRegs + down_regs > kQuarterRegs;
    return r;
}

}  // namespace nvmai
