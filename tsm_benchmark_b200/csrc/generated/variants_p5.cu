// Generated by tsm_benchmark_b200/codegen.py -- do not edit.
// Regenerate with: python -m tsm_benchmark_b200.codegen

#include "../tsm_registry.cuh"

namespace tsm {

extern const Variant kGenPart5[];
const Variant kGenPart5[] = {
    TSM_DMMA_VARIANT("dmma_32x32_t32x32_w8_s3_r128", 32, 32, 4, 4, 8, 3, 128),
    TSM_DMMA_VARIANT("dmma_64x32_t32x32_w8_s3_r80", 64, 32, 4, 4, 8, 3, 80),
    TSM_BULK_VARIANT("bulk_1x1_t1x1_w8_s2_r6144_u1", double, 1, 1, 1, 1, 8, 2, 6144, 1, true, false),
    TSM_BULK_VARIANT("bulk_2x2_t2x2_w8_s4_r1536_u1", double, 2, 2, 2, 2, 8, 4, 1536, 1, true, false),
    TSM_BULK_VARIANT("bulk_4x8_t4x4_w8_s6_r256_u1", double, 4, 8, 4, 4, 8, 6, 256, 1, true, false),
    TSM_BULK_VARIANT("bulk_4x32_t4x8_w8_s6_r64_u1", double, 4, 32, 4, 8, 8, 6, 64, 1, true, false),
    TSM_BULK_VARIANT("bulk_8x8_t4x4_w8_s6_r256_u1", double, 8, 8, 4, 4, 8, 6, 256, 1, true, false),
    TSM_BULK_VARIANT("bulk_8x8_t4x4_w8_s3_r512_u1", double, 8, 8, 4, 4, 8, 3, 512, 1, true, false),
    TSM_BULK_VARIANT("bulk_8x32_t4x8_w8_s3_r192_u1", double, 8, 32, 4, 8, 8, 3, 192, 1, true, false),
    TSM_BULK_VARIANT("bulk_16x8_t8x4_w8_s3_r256_u1", double, 16, 8, 8, 4, 8, 3, 256, 1, true, false),
    TSM_BULK_VARIANT("bulk_16x16_t8x8_w8_s2_r384_u1", double, 16, 16, 8, 8, 8, 2, 384, 1, true, false),
    TSM_BULK_VARIANT("bulk_32x4_t8x4_w8_s2_r192_u1", double, 32, 4, 8, 4, 8, 2, 192, 1, true, false),
    TSM_BULK_VARIANT("bulk_32x16_t8x8_w8_s2_r192_u1", double, 32, 16, 8, 8, 8, 2, 192, 1, true, false),
    TSM_BULK_VARIANT("bulk_64x64_t8x8_w8_s6_r32_u2", double, 64, 64, 8, 8, 8, 6, 32, 2, true, false),
    TSM_BULK_VARIANT("bulk_1x8_t1x4_w8_s6_r384_u1_cap", double, 1, 8, 1, 4, 8, 6, 384, 1, false, false),
    TSM_BULK_VARIANT("bulk_2x16_t2x8_w8_s6_r128_u1_cap", double, 2, 16, 2, 8, 8, 6, 128, 1, false, false),
    TSM_BULK_VARIANT("bulk_4x32_t4x8_w8_s6_r64_u1_cap", double, 4, 32, 4, 8, 8, 6, 64, 1, false, false),
    TSM_BULK_VARIANT("bulk_8x64_t4x8_w8_s6_r48_u1_cap", double, 8, 64, 4, 8, 8, 6, 48, 1, false, false),
    TSM_BULK_VARIANT("bulk_32x1_t8x1_w8_s6_r64_u1_cap", double, 32, 1, 8, 1, 8, 6, 64, 1, false, false),
    TSM_BULK_VARIANT("bulk_64x2_t8x2_w8_s6_r32_u1_cap", double, 64, 2, 8, 2, 8, 6, 32, 1, false, false),
    TSM_DIRECT_VARIANT("direct_1x4_t1x4_th256_cap", double, 1, 4, 1, 4, 256, false),
    TSM_DIRECT_VARIANT("direct_2x8_t2x4_th256_cap", double, 2, 8, 2, 4, 256, false),
    TSM_DIRECT_VARIANT("direct_4x16_t4x8_th256_cap", double, 4, 16, 4, 8, 256, false),
    TSM_DIRECT_VARIANT("direct_8x32_t4x8_th256_cap", double, 8, 32, 4, 8, 256, false),
    TSM_DIRECT_VARIANT("direct_16x64_t8x8_th256_cap", double, 16, 64, 8, 8, 256, false),
    TSM_DIRECT_VARIANT("direct_64x1_t8x1_th256_cap", double, 64, 1, 8, 1, 256, false),
    TSM_BULK_VARIANT("bulkf32_2x2_t2x2_w8_s2_r6144_u1", float, 2, 2, 2, 2, 8, 2, 6144, 1, true, false),
    TSM_BULK_VARIANT("bulkf32_4x4_t4x4_w8_s3_r2048_u1", float, 4, 4, 4, 4, 8, 3, 2048, 1, true, false),
    TSM_BULK_VARIANT("bulkf32_8x8_t4x4_w8_s6_r512_u1", float, 8, 8, 4, 4, 8, 6, 512, 1, true, false),
    TSM_BULK_VARIANT("bulkf32_1x16_t1x8_w8_s6_r384_u1_cap", float, 1, 16, 1, 8, 8, 6, 384, 1, false, false),
    TSM_BULK_VARIANT("bulkf32_2x32_t2x8_w8_s6_r192_u1_cap", float, 2, 32, 2, 8, 8, 6, 192, 1, false, false),
    TSM_BULK_VARIANT("bulkf32_4x64_t4x8_w8_s6_r96_u1_cap", float, 4, 64, 4, 8, 8, 6, 96, 1, false, false),
    TSM_BULK_VARIANT("bulkf32_16x1_t8x1_w8_s6_r384_u1_cap", float, 16, 1, 8, 1, 8, 6, 384, 1, false, false),
    TSM_BULK_VARIANT("bulkf32_32x2_t8x2_w8_s6_r192_u1_cap", float, 32, 2, 8, 2, 8, 6, 192, 1, false, false),
    TSM_BULK_VARIANT("bulkf32_64x4_t8x4_w8_s6_r96_u1_cap", float, 64, 4, 8, 4, 8, 6, 96, 1, false, false),
    TSM_DIRECT_VARIANT("directf32_1x8_t1x4_th256_cap", float, 1, 8, 1, 4, 256, false),
    TSM_DIRECT_VARIANT("directf32_2x16_t2x8_th256_cap", float, 2, 16, 2, 8, 256, false),
    TSM_DIRECT_VARIANT("directf32_4x32_t4x8_th256_cap", float, 4, 32, 4, 8, 256, false),
    TSM_DIRECT_VARIANT("directf32_8x64_t4x8_th256_cap", float, 8, 64, 4, 8, 256, false),
    TSM_DIRECT_VARIANT("directf32_32x1_t8x1_th256_cap", float, 32, 1, 8, 1, 256, false),
    TSM_DIRECT_VARIANT("directf32_64x2_t8x2_th256_cap", float, 64, 2, 8, 2, 256, false),
    TSM_GRAM_DMMA_VARIANT("dmma_48x48_gram_w8_s3_r160", 48, 8, 3, 160),
    TSM_BULK_VARIANT("bulk_4x4_t4x4_w8_s3_r2048_u1_gram", double, 4, 4, 4, 4, 8, 3, 2048, 1, true, true),
    TSM_DMMA_VARIANT("dmma_32x32_t32x32_w8_s4_r96", 32, 32, 4, 4, 8, 4, 96),
    TSM_DMMA_VARIANT("dmma_32x32_t32x32_w12_s2_r192", 32, 32, 4, 4, 12, 2, 192),
    TSM_GRAM_DMMA_VARIANT("dmma_64x64_gram_w12_s2_r192", 64, 12, 2, 192),
    TSM_TILE_VARIANT("direct_dmma_32x16_cap", double, 32, 16),
    TSM_TILE_VARIANT("direct_dmma_48x8_cap", double, 48, 8),
    TSM_TILE_VARIANT("direct_dmma_56x24_cap", double, 56, 24),
    TSM_TILE_VARIANT("direct_dmma_64x32_cap", double, 64, 32),
    TSM_TILE_VARIANT("directf32_dmma_24x8_cap", float, 24, 8),
    TSM_TILE_VARIANT("directf32_dmma_40x16_cap", float, 40, 16),
    TSM_TILE_VARIANT("directf32_dmma_48x40_cap", float, 48, 40),
    TSM_TILE_VARIANT("directf32_dmma_56x56_cap", float, 56, 56),
    TSM_TILE_VARIANT("directf32_dmma_64x64_cap", float, 64, 64),
};
extern const int kGenPart5Count;
const int kGenPart5Count = 55;

}  // namespace tsm
