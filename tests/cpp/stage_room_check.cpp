// The rule of stage_room.h, by the shared memory and registers that the decode stages really take: what it promises holds, and
// it does not hang on the bit width of the codes.
#include <cstdio>

#include "../../nvmai_b200/csrc/stage_room.h"

using namespace nvmai;

int main() {
    int bad = 0;
    auto expect = [&](const char *what, bool ok) { if (!ok) { std::printf("%s\n", what); ++bad; } };
    const uint32_t sms = 148;
    // (shared memory of a block of stage 2 and 3, their blocks, warps of a block of stage 3)
    StageRoom r = stage_room(44864, 66816, 288, 128, sms, 18, true);            // 2048 / 512, 4-bit
    expect("4-bit 2048 / 512", r.whole_shared && r.early && r.lean);
    r = stage_room(40768, 103680, 288, 64, sms, 18, true);                      // 1024 / 512, 8-bit: the same room, the same cap
    expect("8-bit 1024 / 512", r.whole_shared && r.early && r.lean);
    r = stage_room(44864, 60416, 256, 128, sms, 16, true);                      // top-7 and a shared expert: 16 warps fit at 64
    expect("16 warps", r.early && !r.lean);
    r = stage_room(44864, 122112, 576, 128, sms, 18, true);                     // 2048 / 1024, 4-bit: four blocks an SM leave no room
    expect("4-bit 2048 / 1024", !r.whole_shared && !r.early && !r.lean && r.beside_two);
    r = stage_room(85824, 122112, 576, 256, sms, 18, true);                     // 4096 / 1024, 4-bit
    expect("4-bit 4096 / 1024", !r.whole_shared && !r.early && !r.lean && !r.beside_two);
    r = stage_room(44864, 29952, 72, 128, sms, 18, true);                       // a block an SM
    expect("2048 / 128", r.early && !r.lean);
    r = stage_room(44864, 39168, 288, 256, sms, 18, true);                      // two rows of 2048 / 256: half of stage 3 could be early
    expect("two rows", r.early && !r.lean);
    r = stage_room(77632, 58368, 320, 256, sms, 10, true);                      // 8-bit, top-4, two rows: an SM holds two blocks, not three
    expect("two by shared memory", r.whole_shared && !r.lean);
    r = stage_room(44864, 37888, 320, 256, sms, 10, true);                      // 4-bit: three
    expect("three", r.whole_shared && r.lean);
    r = stage_room(44864, 66816, 0, 0, 0, 18, true);                            // a device that was not asked
    expect("no device", !r.whole_shared && !r.early && !r.lean);
    for (size_t gate_up = 8192; gate_up <= 160 * 1024; gate_up += 4096)
        for (size_t down = 8192; down <= 200 * 1024; down += 8192)
            for (uint32_t blocks = 1; blocks <= 1200; blocks += 29)
                for (uint32_t warps = 2; warps <= 18; warps += 2) {
                    r = stage_room(gate_up, down, blocks, 128, sms, warps, true);
                    const uint32_t most = (blocks + sms - 1) / sms, down_regs = (warps + 3) / 4 * 32 * 56;
                    // every SM that holds two blocks of stage 2 or fewer has room for one of stage 3
                    const uint32_t n = most < 2 ? most : 2;
                    if (r.early && most <= 2)
                        expect("early without room", n * (gate_up + 1024) + down + 1024 <= 228 * 1024 &&
                                                         n * 2 * 32 * (r.lean ? 56 : 64) + down_regs <= 16384);
                    expect("cap without use", !r.lean || r.whole_shared);
                    expect("early only where it fits", !r.early || r.whole_shared);
                    // row copies never start early
                    const StageRoom rows = stage_room(gate_up, down, blocks, 128, sms, warps, false);
                    expect("row copies", !rows.early && !rows.lean && (!rows.whole_shared || blocks > sms));
                }
    std::printf(bad ? "FAILED %d\n" : "PASSED\n", bad);
    return bad != 0;
}
