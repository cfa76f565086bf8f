// launch_pcg_amg for systems of three sizes on two devices in turn, linked with
// fake_cudart.cpp; with an argument, the second device takes no cluster of more
// than 8 blocks.
#include "pg_device.cuh"

extern int fake_device, fake_largest[2];

namespace pg {
int sm_count() { return 152; }
void count_launches(int) {}
}  // namespace pg

int main(int argc, char **) {
    if (argc > 1) fake_largest[1] = 8;
    pg::PcgArgs a{};
    pg::AmgDev m{};
    for (int d : {0, 1, 0, 1}) {
        fake_device = d;
        for (int n : {400, 12288, 12289}) {
            a.n = n;
            if (pg::launch_pcg_amg(a, m, nullptr) != 0) return 1;
        }
    }
    return 0;
}
