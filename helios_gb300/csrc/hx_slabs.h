// Slabs of triples for the (T) correction (host code): how many fit.
#pragma once

struct SlabPlan {
    bool keep;               // the terms' operands are sliced once per slab and stay for all twelve
    long long triples;       // most triples of a slab; fewer than o: not even a row (i, j) fits
    double bytes;            // memory of the integrals and one row of triples in that form
};

// A slab holds W (v^3 doubles per triple) and the 7-slice bf16 copies of the
// operand that a k-batched term slices per triple (v^2 x v, 14 B per
// element), within half of what the integrals leave of the free memory and
// 24 GB. Where the slices of every term's operands fit beside it they are made
// once per slab (the estimate counts (bd|ai), (ck|jl) and t2 twice over
// for their views); else the terms slice theirs one after the other into the
// same scratch, so that a row needs no more than W and one term's slices.
inline SlabPlan plan_slabs(int N, int o, int v, double free_bytes)
{
    const double vv = (double)v * v, ov = (double)o * v, kv = (v + 7) / 8 * 8;
    const double I1 = ov * vv, J = ov * o * o, per = 8.0 * vv * v + 14.0 * vv * kv;
    const double integrals = 8.0 * (I1 + J + N * vv + 2.0 * N * (double)o * o);
    const double slices = 28.0 * (2.0 * I1 + 4.0 * J + 6.0 * ov * ov);
    SlabPlan p{};
    for (int keep = 1; keep >= 0; --keep) {
        const double fixed = integrals + (keep ? slices : 0.0), half = 0.5 * (free_bytes - fixed);
        p = {keep == 1, (long long)((half < 24e9 ? half : 24e9) / per), fixed + o * per};
        if (p.triples >= o) break;
    }
    return p;
}
