// Reads the L2's size and cavities' sizes (ended by 0), prints the first cavity of
// every group, their number and the cost of the cut (partition.h).  Built and run
// by tests/test_batch_partition_cpu.py.
#include <cstdio>
#include "partition.h"
int main() {
    unsigned long long l2, b;
    while (std::scanf("%llu", &l2) == 1) {
        std::vector<size_t> bytes;
        while (std::scanf("%llu", &b) == 1 && b) bytes.push_back(size_t(b));
        const std::vector<int> first = cav::partition_groups(bytes, size_t(l2));
        double cost = 0.0;
        for (size_t g = 0; g + 1 < first.size(); ++g) {
            double sum = 0.0;
            for (int i = first[g]; i < first[g + 1]; ++i) sum += double(bytes[i]);
            cost += cav::group_cost(sum, double(l2));
        }
        for (int i : first) std::printf("%d ", i);
        std::printf("%.17g\n", cost);
    }
}
