// Host test of lbm_b200/csrc/sweep_rules.hpp: whatever box the rules are asked
// about, the pass that they choose is one that the device can launch.  Exit
// code 0 on success.
#include <cstdio>
#include <initializer_list>

#include "../../lbm_b200/csrc/sweep_rules.hpp"

namespace {

bool launchable(int lx, int ly, int lz, int tx, int ty, int zlen)
{
    const long long gx = (lx + tx - 1LL) / tx, gy = (ly + ty - 1LL) / ty, gz = (lz + zlen - 1LL) / zlen;
    return zlen >= 1 && zlen <= lz && gx <= 0x7fffffffLL && gy <= 65535 && gz <= 65535;
}

struct Box {
    int lx, ly, lz;
    bool passes;
};

}  // namespace

int main()
{
    using namespace lbm;
    // boxes the rules sent to passes whose tile rows no grid holds
    if (fp64_pass_zlen(28, 400000, 3, 148) != 0 || fp64_pass_zlen(30, 400000, 11, 148) != 0) return 1;
    // the last row count that fits and the first that does not
    if (!fp64_pass_fits(6 * 65535, 6 * 65535) || fp64_pass_fits(6 * 65535 + 1, 6 * 65535 + 1)) return 2;
    if (!mixed_pass_fits(8 * 65535, 8 * 65535) || mixed_pass_fits(8 * 65535 + 1, 8 * 65535 + 1)) return 3;
    if (fp64_pass_fits(1, 143165577) || !fp64_pass_fits(1, 143165576)) return 4;
    // correction sweeps of the refinement form: passes where they were measured 3 % or
    // more faster, single sweeps where those were, whatever the plain sweeps take
    for (const auto& b : {Box{88, 88, 88, true}, Box{128, 47, 100, true}, Box{96, 96, 96, true}, Box{118, 143, 129, true},
                          Box{191, 141, 69, true}, Box{160, 160, 160, true}, Box{45, 183, 190, true}, Box{110, 57, 131, true}, Box{25, 161, 182, true}, Box{136, 98, 177, false}, Box{156, 88, 48, false},
                          Box{64, 64, 64, false}, Box{130, 34, 150, false}, Box{33, 150, 150, false}})
        if ((mixed_pass(b.lx, b.ly, b.lz, 148).refine_zlen > 0) != b.passes) return 9;
    const int extents[] = {1, 2, 3, 5, 6, 7, 8, 9, 16, 30, 31, 32, 33, 47, 64, 75, 96, 131, 203, 256, 1000, 65535, 393210, 393211,
                           524280, 524281, 4000000};
    long long chosen = 0;
    for (int lx : extents)
        for (int ly : extents)
            for (int lz : extents) {
                if (lx < 2 || lz > 65535) continue;   // no such box
                if (static_cast<long long>(lx) * ly * lz > 400000000LL) continue;
                for (int sms : {1, 132, 148, 160}) {
                    const int z64 = fp64_pass_zlen(lx, ly, lz, sms);
                    if (z64 && !launchable(lx, ly, lz, F2_TX, F2_TY, z64)) return 5;
                    const MixedPass m = mixed_pass(lx, ly, lz, sms);
                    if (m.zlen && !launchable(lx, ly, lz, S2_TX, m.tall ? S2_TALL : S2_TY, m.zlen)) return 6;
                    if (m.refine_zlen && !launchable(lx, ly, lz, S2_TX, S2_TALL, m.refine_zlen)) return 7;
                    chosen += (z64 > 0) + (m.zlen > 0);
                }
            }
    if (chosen < 1000) return 8;
    std::puts("sweep rules ok");
    return 0;
}
