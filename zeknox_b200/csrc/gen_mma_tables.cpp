// gen_mma_tables.cpp -- build step: writes the tables of mma_tables.h as C
// initialiser lists (one macro per hash) to standard output.
#include <stdio.h>

#include "mma_tables.h"

static void print_tables(const char *name, const zk::MmaTables &t)
{
    for (int d = 0; d < 3; d++) printf("#define ZK_MMA_%s_H%d 0x%016llxULL\n", name, d + 1, (unsigned long long)t.h[d]);
    printf("#define ZK_MMA_%s_LIST \\\n", name);
    for (size_t i = 0; i < t.w.size(); i++)
        printf("0x%x,%s", t.w[i], i + 1 == t.w.size() ? "\n" : i % 16 == 15 ? " \\\n" : "");
}

int main()
{
    printf("// written by gen_mma_tables.cpp\n#pragma once\n");
    static const uint64_t rc[360] = {ZK_POSEIDON_RC_LIST};
    printf("#define ZK_MMA_POSEIDON_RC0");
    for (int i = 0; i < 12; i++) printf(" 0x%016llxULL%s", (unsigned long long)rc[i], i < 11 ? "," : "\n");
    print_tables("POSEIDON", zk::make_mma_tables(0));
    print_tables("POSEIDON2", zk::make_mma_tables(3));
    print_tables("MONOLITH", zk::make_mma_monolith());
    return 0;
}
