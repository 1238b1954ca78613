// Prints the kernel that matmul_noalloc picks:  matmul_pick columns k rows SMs values_a_load
#include "../../aspen_b200/csrc/matmul_pick.h"
#include <cstdio>
#include <cstdlib>

int main(int, char **argv) {
    unsigned a[5];
    for (int i = 0; i < 5; i++) a[i] = (unsigned)atoi(argv[i + 1]);
    const char *name[] = {"fma 128x64", "fma 64x64", "fma 32x32", "split 128", "split 64"};
    printf("%s", name[pick_matmul(a[0], a[1], a[2], a[3], (int)a[4])]);
    return 0;
}
