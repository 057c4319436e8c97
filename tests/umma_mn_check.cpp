// Host check of the GEMM's transposed operand stages (elanfmt_gb300/csrc/ewf_umma.h), compiled with
// g++ by tests/test_umma_mn_layout_cpu.py: what the TMA boxes of 64 rows x BK deliver under the
// 128-byte swizzle is where the tensor core's canonical MN-major SWIZZLE_128B layout, with the
// descriptor's offsets, looks for it, and no MMA of a stage reads outside its operand.
#include <cstdio>

#include "ewf_umma.h"

using namespace ewf_umma;

int main()
{
    for (int rows = 64; rows <= 128; rows += 64) {
        for (int j = 0; j < BK / MMA_K; ++j) {
            const uint64_t d = smem_desc_sw128_mn(0x2A400 + j * MN_K_STEP);
            const uint32_t start = (uint32_t)(d & 0x3FFF) << 4, lbo = (uint32_t)((d >> 16) & 0x3FFF) << 4, sbo = (uint32_t)((d >> 32) & 0x3FFF) << 4;
            if (start != 0x2A400u + j * MN_K_STEP || ((d >> 46) & 3) != 1 || (d >> 61) != (uint64_t)LAYOUT_SW128) return printf("FAIL fields\n"), 1;
            for (int mn = 0; mn < rows; ++mn)
                for (int kk = 0; kk < MMA_K; ++kk) {
                    // ((T,8,m),(8,k)) : ((1,T,LBO),(8T,SBO)) in 16-byte units of T = 8 elements, then the swizzle on address bits
                    uint32_t a = start + (mn % 64) * 2 + (mn / 64) * lbo + (kk % 8) * 128 + (kk / 8) * sbo;
                    a ^= ((a >> 7) & 7) << 4;
                    const int k = j * MMA_K + kk;
                    // the TMA box of block mn / 64: row k holds 64 values, 16-byte chunk c at c ^ (k % 8)
                    const uint32_t want = 0x2A400u + (mn / 64) * MN_BLOCK_BYTES + k * 128 + ((((mn % 64) * 2 / 16) ^ (k % 8)) * 16) + (mn * 2) % 16;
                    if (a != want || want != 0x2A400u + mn_offset(mn, k)) return printf("FAIL %d %d %d\n", rows, mn, k), 1;
                    if (a + 2 > 0x2A400u + (uint32_t)rows * ROW_BYTES) return printf("FAIL range\n"), 1;
                }
        }
        if (rows / MN_ATOM * MN_BLOCK_BYTES != b_bytes(rows)) return printf("FAIL bytes\n"), 1;
    }
    const uint32_t id = instr_desc_bf16_f32(BM, 64, true, true);
    if (((id >> 15) & 3) != 3 || (id & ~(3u << 15)) != instr_desc_bf16_f32(BM, 64)) return printf("FAIL idesc\n"), 1;
    printf("ok\n");
    return 0;
}
