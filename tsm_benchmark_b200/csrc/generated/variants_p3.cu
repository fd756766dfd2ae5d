// Generated by tsm_benchmark_b200/codegen.py -- do not edit.
// Regenerate with: python -m tsm_benchmark_b200.codegen

#include "../tsm_registry.cuh"

namespace tsm {

extern const Variant kGenPart3[];
const Variant kGenPart3[] = {
    TSM_DMMA_VARIANT("dmma_16x64_t16x64_w8_s3_r96", 16, 64, 2, 8, 8, 3, 96),
    TSM_DMMA_VARIANT("dmma_48x64_t16x64_w9_s3_r72", 48, 64, 2, 8, 9, 3, 72),
    TSM_BULK_VARIANT("bulk_1x1_t1x1_w8_s3_r4096_u1", double, 1, 1, 1, 1, 8, 3, 4096, 1, true, false),
    TSM_BULK_VARIANT("bulk_2x2_t2x2_w8_s6_r1024_u2", double, 2, 2, 2, 2, 8, 6, 1024, 2, true, false),
    TSM_BULK_VARIANT("bulk_4x4_t4x4_w8_s4_r768_u1", double, 4, 4, 4, 4, 8, 4, 768, 1, true, false),
    TSM_BULK_VARIANT("bulk_4x16_t4x8_w8_s4_r128_u1", double, 4, 16, 4, 8, 8, 4, 128, 1, true, false),
    TSM_BULK_VARIANT("bulk_8x4_t4x4_w8_s4_r384_u1", double, 8, 4, 4, 4, 8, 4, 384, 1, true, false),
    TSM_BULK_VARIANT("bulk_8x8_t2x8_w8_s10_r128_u1", double, 8, 8, 2, 8, 8, 10, 128, 1, true, false),
    TSM_BULK_VARIANT("bulk_8x16_t4x8_w8_s2_r384_u1", double, 8, 16, 4, 8, 8, 2, 384, 1, true, false),
    TSM_BULK_VARIANT("bulk_16x4_t8x4_w8_s2_r384_u1", double, 16, 4, 8, 4, 8, 2, 384, 1, true, false),
    TSM_BULK_VARIANT("bulk_16x16_t8x8_w8_s3_r256_u1", double, 16, 16, 8, 8, 8, 3, 256, 1, true, false),
    TSM_BULK_VARIANT("bulk_32x4_t8x4_w8_s3_r128_u1", double, 32, 4, 8, 4, 8, 3, 128, 1, true, false),
    TSM_BULK_VARIANT("bulk_32x16_t8x8_w8_s3_r128_u1", double, 32, 16, 8, 8, 8, 3, 128, 1, true, false),
    TSM_BULK_VARIANT("bulk_32x32_t8x8_w8_s2_r192_u1", double, 32, 32, 8, 8, 8, 2, 192, 1, true, false),
    TSM_BULK_VARIANT("bulk_1x2_t1x2_w8_s6_r1280_u1_cap", double, 1, 2, 1, 2, 8, 6, 1280, 1, false, false),
    TSM_BULK_VARIANT("bulk_2x4_t2x4_w8_s6_r512_u1_cap", double, 2, 4, 2, 4, 8, 6, 512, 1, false, false),
    TSM_BULK_VARIANT("bulk_4x8_t4x4_w8_s6_r256_u1_cap", double, 4, 8, 4, 4, 8, 6, 256, 1, false, false),
    TSM_BULK_VARIANT("bulk_8x16_t4x8_w8_s6_r128_u1_cap", double, 8, 16, 4, 8, 8, 6, 128, 1, false, false),
    TSM_BULK_VARIANT("bulk_16x32_t8x8_w8_s6_r64_u1_cap", double, 16, 32, 8, 8, 8, 6, 64, 1, false, false),
    TSM_BULK_VARIANT("bulk_32x64_t8x8_w8_s6_r40_u1_cap", double, 32, 64, 8, 8, 8, 6, 40, 1, false, false),
    TSM_DIRECT_VARIANT("direct_1x1_t1x1_th256_cap", double, 1, 1, 1, 1, 256, false),
    TSM_DIRECT_VARIANT("direct_2x2_t2x2_th256_cap", double, 2, 2, 2, 2, 256, false),
    TSM_DIRECT_VARIANT("direct_4x4_t4x4_th256_cap", double, 4, 4, 4, 4, 256, false),
    TSM_DIRECT_VARIANT("direct_8x8_t4x4_th256_cap", double, 8, 8, 4, 4, 256, false),
    TSM_DIRECT_VARIANT("direct_16x16_t8x8_th256_cap", double, 16, 16, 8, 8, 256, false),
    TSM_DIRECT_VARIANT("direct_32x32_t8x8_th256_cap", double, 32, 32, 8, 8, 256, false),
    TSM_DIRECT_VARIANT("direct_64x64_t8x8_th256_cap", double, 64, 64, 8, 8, 256, false),
    TSM_BULK_VARIANT("bulkf32_1x1_t1x1_w8_s3_r8192_u1", float, 1, 1, 1, 1, 8, 3, 8192, 1, true, false),
    TSM_BULK_VARIANT("bulkf32_2x2_t2x2_w8_s6_r2048_u1", float, 2, 2, 2, 2, 8, 6, 2048, 1, true, false),
    TSM_BULK_VARIANT("bulkf32_1x4_t1x4_w8_s6_r1536_u1_cap", float, 1, 4, 1, 4, 8, 6, 1536, 1, false, false),
    TSM_BULK_VARIANT("bulkf32_2x8_t2x4_w8_s6_r768_u1_cap", float, 2, 8, 2, 4, 8, 6, 768, 1, false, false),
    TSM_BULK_VARIANT("bulkf32_4x16_t4x8_w8_s6_r384_u1_cap", float, 4, 16, 4, 8, 8, 6, 384, 1, false, false),
    TSM_BULK_VARIANT("bulkf32_8x32_t4x8_w8_s6_r192_u1_cap", float, 8, 32, 4, 8, 8, 6, 192, 1, false, false),
    TSM_BULK_VARIANT("bulkf32_16x64_t8x8_w8_s6_r96_u1_cap", float, 16, 64, 8, 8, 8, 6, 96, 1, false, false),
    TSM_BULK_VARIANT("bulkf32_64x1_t8x1_w8_s6_r96_u1_cap", float, 64, 1, 8, 1, 8, 6, 96, 1, false, false),
    TSM_DIRECT_VARIANT("directf32_1x2_t1x2_th256_cap", float, 1, 2, 1, 2, 256, false),
    TSM_DIRECT_VARIANT("directf32_2x4_t2x4_th256_cap", float, 2, 4, 2, 4, 256, false),
    TSM_DIRECT_VARIANT("directf32_4x8_t4x4_th256_cap", float, 4, 8, 4, 4, 256, false),
    TSM_DIRECT_VARIANT("directf32_8x16_t4x8_th256_cap", float, 8, 16, 4, 8, 256, false),
    TSM_DIRECT_VARIANT("directf32_16x32_t8x8_th256_cap", float, 16, 32, 8, 8, 256, false),
    TSM_DIRECT_VARIANT("directf32_32x64_t8x8_th256_cap", float, 32, 64, 8, 8, 256, false),
    TSM_GRAM_DMMA_VARIANT("dmma_16x16_gram_w8_s4_r256", 16, 8, 4, 256),
    TSM_BULK_VARIANT("bulk_1x1_t1x1_w8_s3_r8192_u1_gram", double, 1, 1, 1, 1, 8, 3, 8192, 1, true, true),
    TSM_DMMA_VARIANT("dmma_16x16_t16x16_w8_s4_r192", 16, 16, 2, 2, 8, 4, 192),
    TSM_GRAM_DMMA_VARIANT("dmma_16x16_gram_w8_s3_r512", 16, 8, 3, 512),
    TSM_GRAM_DMMA_VARIANT("dmma_64x64_gram_w8_s2_r192", 64, 8, 2, 192),
    TSM_TILE_VARIANT("direct_dmma_24x24_cap", double, 24, 24),
    TSM_TILE_VARIANT("direct_dmma_40x32_cap", double, 40, 32),
    TSM_TILE_VARIANT("direct_dmma_56x8_cap", double, 56, 8),
    TSM_TILE_VARIANT("direct_dmma_64x16_cap", double, 64, 16),
    TSM_TILE_VARIANT("directf32_dmma_16x8_cap", float, 16, 8),
    TSM_TILE_VARIANT("directf32_dmma_32x32_cap", float, 32, 32),
    TSM_TILE_VARIANT("directf32_dmma_48x24_cap", float, 48, 24),
    TSM_TILE_VARIANT("directf32_dmma_56x40_cap", float, 56, 40),
    TSM_TILE_VARIANT("directf32_dmma_64x48_cap", float, 64, 48),
};
extern const int kGenPart3Count;
const int kGenPart3Count = 55;

}  // namespace tsm
