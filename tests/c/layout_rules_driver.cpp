// The layout rules (layout_rules.h) for tests without a GPU.
#include "layout_rules.h"

extern "C" int rule_lanes(long n, double avg, long groups, int lean, long fused_rows, int asked) {
    return layout::lanes_for_shape(n, avg, groups, lean != 0, fused_rows, asked);
}

extern "C" int rule_fused(int acol, int a, int r, int p) { return layout::fused_layouts(acol, a, r, p) ? 1 : 0; }
