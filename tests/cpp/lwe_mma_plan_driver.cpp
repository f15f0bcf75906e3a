// Prints lwe_mma_plan's rows, rows_pad, splits, plane_bytes and part_bytes for argument tuples
// "planes kpad width batch sms" read from stdin. Used by tests/test_lwe_mma_plan_cpu.py (no GPU).
#include <cstdint>
#include <iostream>

#include "lwe_mma_plan.h"

int main() {
    int planes;
    uint32_t kpad, width;
    uint64_t batch, sms;
    while (std::cin >> planes >> kpad >> width >> batch >> sms) {
        const tp::LweMmaPlan p = tp::lwe_mma_plan(planes, kpad, width, batch, sms);
        std::cout << p.rows << " " << p.rows_pad << " " << p.splits << " " << p.plane_bytes << " " << p.part_bytes << " "
                  << tp::lwe_mma_fits(planes, width) << "\n";
    }
    return 0;
}
