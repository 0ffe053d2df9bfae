// Host-side check of the MN-major operands in sph_tcgen05.cuh against CuTe's own construction
// (cute/atom/mma_traits_sm100.hpp): the layout of 8-element groups, the descriptor strides and
// the instruction descriptors.  Prints "ok" and exits 0 when everything agrees.
#include <cstdio>
#include <cute/tensor.hpp>
#include <cute/atom/mma_traits_sm100.hpp>
#include "sph_tcgen05.cuh"

using namespace cute;

// An MN-major operand of R x K elements whose groups of 8 along R are MNG elements apart and those
// along K KG elements apart, as the kernels index it, against CuTe's atom over the same strides.
template <int R, int MNG, int KG>
static int check_operand(const char* name) {
    int bad = 0;
    auto L = make_layout(make_shape(make_shape(Int<8>{}, Int<R / 8>{}), make_shape(Int<8>{}, Int<2>{})),
                         make_stride(make_stride(Int<1>{}, Int<MNG>{}), make_stride(Int<8>{}, Int<KG>{})));
    UMMA::SmemDescriptor d = UMMA::make_umma_desc<UMMA::Major::MN>(make_tensor(make_smem_ptr((bfloat16_t*)nullptr), L));
    const uint64_t mine = wsph::umma_desc_mnmajor(0u, KG * 2, MNG * 2), theirs = static_cast<uint64_t>(d) & ~0x3FFFull;
    if (mine != theirs) {
        std::printf("%s: descriptor %016llx, CuTe %016llx\n", name, (unsigned long long)mine, (unsigned long long)theirs);
        ++bad;
    }
    return bad;
}

int main() {
    int bad = 0;
    // one k-step of the activations: 64, 72 or 16 units x 16 samples, chunks of 8 units x 128 samples
    bad += check_operand<64, 8 * 128, 64>("dZ, 64 units");
    bad += check_operand<72, 8 * 128, 64>("H and ones, 72 units");
    bad += check_operand<16, 8 * 128, 64>("X and ones, 16 units");
    // one k-step of W read as its transpose: 64 inputs x 16 outputs of the K-major [64 out x K in] copy
    bad += check_operand<64, 8 * 64, 64>("W^T");
    for (int i = 0; i < 64; ++i)
        for (int o = 0; o < 64; ++o)
            if (wsph::umma_k_index(o, i, 64) != (i / 8) * 512 + i % 8 + (o / 8) * 64 + (o % 8) * 8) ++bad;
    const uint32_t g = static_cast<uint32_t>(UMMA::make_instr_desc<bfloat16_t, bfloat16_t, float, 64, 72, UMMA::Major::MN, UMMA::Major::MN>());
    const uint32_t g1 = static_cast<uint32_t>(UMMA::make_instr_desc<bfloat16_t, bfloat16_t, float, 64, 16, UMMA::Major::MN, UMMA::Major::MN>());
    const uint32_t dh = static_cast<uint32_t>(UMMA::make_instr_desc<bfloat16_t, bfloat16_t, float, 128, 64, UMMA::Major::K, UMMA::Major::MN>());
    if (g != wsph::umma_idesc_bf16_f32<64, 72, true, true>() || g1 != wsph::umma_idesc_bf16_f32<64, 16, true, true>() || dh != wsph::umma_idesc_bf16_f32<128, 64, false, true>()) {
        std::printf("instruction descriptors: CuTe %08x %08x %08x\n", g, g1, dh);
        ++bad;
    }
    std::printf(bad ? "mismatch\n" : "ok\n");
    return bad ? 1 : 0;
}
