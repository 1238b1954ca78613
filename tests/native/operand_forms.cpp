// Prints, for each layer of a cfg (and a sequence length), how its operands reach the tensor cores (0: they do not).
#include "../../aspen_b200/csrc/internal.h"

int main(int, char **argv) {
    aspen_dnn_t *dnn = apu_create_dnn(argv[1], nullptr);
    if (!dnn) return 1;
    for (const aspen_layer_t &l : dnn->layers) {
        const OperandForm f = operand_form(&l, (unsigned)atoi(argv[2]));
        printf("%s %u %u %u\n", layer_type_str[l.type], f.kind, f.image ? 1u : 0u, f.kind == 2 ? f.k() : 0u);
    }
    apu_destroy_dnn(dnn);
    return 0;
}
