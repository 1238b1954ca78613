// Builds a tile graph (cfg, batch, file to save it in) while pthread_create fails from the N-th call on: few_threads N cfg batch file
#include "../../include/aspen_b200.h"

#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <cstdlib>

static int g_left = 0;

extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
    if (--g_left <= 0) return EAGAIN;
    static auto real = (int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *))dlsym(RTLD_NEXT, "pthread_create");
    return real(t, a, f, arg);
}

int main(int, char **argv) {
    g_left = atoi(argv[1]);
    aspen_dnn_t *dnn = apu_create_dnn(argv[2], nullptr);
    nasm_t *nasm = dnn ? apu_create_nasm(dnn, 100, (unsigned)atoi(argv[3])) : nullptr;
    if (!nasm) return 1;
    apu_save_nasm_to_file(nasm, argv[4]);
    apu_destroy_nasm(nasm);
    apu_destroy_dnn(dnn);
    return 0;
}
