// The layout rules (layout_rules.h) for tests without a GPU.
#include "layout_rules.h"

extern "C" int rule_lanes(long n, int rows, const int* ptr, long groups, int lean, long fused_rows, int asked) {
    return layout::lanes_for(n, rows, ptr, groups, lean != 0, fused_rows, asked);
}

extern "C" int rule_lanes64(int rows, const int* ptr, int lanes) {
    return layout::lanes64_for(layout::row_counts(rows, ptr), lanes);
}

extern "C" int rule_fused(int acol, int a, int r, int p) { return layout::fused_layouts(acol, a, r, p) ? 1 : 0; }

extern "C" int rule_stage_lanes(const int* len, int count, int lanes, int asked) {
    return layout::stage_lanes64(std::vector<int>(len, len + count), lanes, asked);
}

extern "C" int rule_groups_allowed(int asked) { return layout::groups_allowed(asked) ? 1 : 0; }

extern "C" int rule_sell_variant(int f64, int long_rows, long npos) {
    return (int)layout::sell_variant(f64 != 0, long_rows != 0, npos);
}

extern "C" int rule_lean_images(long rows, long c, long p, long e) { return layout::lean_images(rows, c, p, e) ? 1 : 0; }

extern "C" int rule_seg_chunk(int n, int lean) { return layout::seg_chunk(n, lean != 0); }
