// sl8_dispatch_table.h -- GENERATED by `python -m siglip_b200.sweep --emit-table siglip_b200/sweeps/b200.csv`.
// One row per (layer, N, K, smallest M) -> kernel variant, from the sweep on B200; pick_variant() takes the
// row with the largest m_min <= M for an exact (layer, N, K) match and asks its cost model otherwise.
#pragma once

struct Sl8DispatchRow { int op; int n; int k; long long m_min; int variant; };

static const Sl8DispatchRow kSl8DispatchTable[] = {
    {SL8_OP_PATCH_EMBED, 768, 768, 0LL, 20},
    {SL8_OP_PATCH_EMBED, 768, 768, 1568LL, 18},
    {SL8_OP_PATCH_EMBED, 768, 768, 12544LL, 17},
    {SL8_OP_PATCH_EMBED, 768, 768, 50176LL, 5},
    {SL8_OP_PATCH_EMBED, 1152, 588, 0LL, 20},
    {SL8_OP_PATCH_EMBED, 1152, 588, 1458LL, 18},
    {SL8_OP_PATCH_EMBED, 1152, 588, 2187LL, 20},
    {SL8_OP_PATCH_EMBED, 1152, 588, 3645LL, 18},
    {SL8_OP_PATCH_EMBED, 1152, 588, 4374LL, 21},
    {SL8_OP_PATCH_EMBED, 1152, 588, 7290LL, 17},
    {SL8_OP_PATCH_EMBED, 1152, 588, 8748LL, 21},
    {SL8_OP_PATCH_EMBED, 1152, 588, 10206LL, 17},
    {SL8_OP_PATCH_EMBED, 1152, 588, 11664LL, 21},
    {SL8_OP_PATCH_EMBED, 1152, 588, 23328LL, 17},
    {SL8_OP_FC1_GELU, 3072, 768, 0LL, 20},
    {SL8_OP_FC1_GELU, 3072, 768, 490LL, 18},
    {SL8_OP_FC1_GELU, 3072, 768, 6272LL, 14},
    {SL8_OP_FC1_GELU, 4304, 1152, 0LL, 18},
    {SL8_OP_FC1_GELU, 4304, 1152, 2551LL, 19},
    {SL8_OP_FC1_GELU, 4304, 1152, 2916LL, 15},
    {SL8_OP_FC2_RESIDUAL, 768, 3072, 0LL, 20},
    {SL8_OP_FC2_RESIDUAL, 768, 3072, 1568LL, 6},
    {SL8_OP_FC2_RESIDUAL, 768, 3072, 3136LL, 21},
    {SL8_OP_FC2_RESIDUAL, 768, 3072, 12544LL, 1},
    {SL8_OP_FC2_RESIDUAL, 1152, 4304, 0LL, 20},
    {SL8_OP_FC2_RESIDUAL, 1152, 4304, 1093LL, 19},
    {SL8_OP_FC2_RESIDUAL, 1152, 4304, 1822LL, 6},
    {SL8_OP_FC2_RESIDUAL, 1152, 4304, 2187LL, 21},
    {SL8_OP_FC2_RESIDUAL, 1152, 4304, 3645LL, 7},
    {SL8_OP_FC2_RESIDUAL, 1152, 4304, 4374LL, 21},
    {SL8_OP_FC2_RESIDUAL, 1152, 4304, 7290LL, 1},
    {SL8_OP_FC2_RESIDUAL, 1152, 4304, 8748LL, 21},
};
static const int kSl8DispatchRows = 32;
