// Prints the tile rows, columns and number of each layer of a cfg's device plan in tensor-core mode: plan_tiles cfg batch seq sms
#include "../../aspen_b200/csrc/internal.h"

int main(int, char **argv) {
    aspen_dnn_t *dnn = apu_create_dnn(argv[1], nullptr);
    nasm_t *nasm = dnn ? apu_create_transformer_nasm(dnn, 100, (unsigned)atoi(argv[2]), (unsigned)atoi(argv[3])) : nullptr;
    nasm_t *plan = nasm ? plan_device_tiles(nasm, 0, (unsigned)atoi(argv[4]), false) : nullptr;
    if (!plan) return 1;
    for (const nasm_ldata_t &ld : plan->ldata) printf("%s %u %u %u\n", layer_type_str[ld.layer->type], ld.ninst_tile_dims[OUT_H], ld.ninst_tile_dims[OUT_W], ld.num_ninst);
    delete plan;
    apu_destroy_nasm(nasm);
    apu_destroy_dnn(dnn);
    return 0;
}
