"""Generates treelet_dp_unrolled.cuh: the LBVH+ subset DP for N = 4..7 treelet leaves as
straight-line code, so that every subset cost lives in a register.

The DP is the one of optimizeTreeletSerial (src/cuda/lbvh_plus_builder.cu:119-165): subsets in
increasing numeric order (every proper subset comes first); cost[s] = min over splits of
cost[p] + cost[s ^ p], plus the area of s; single leaves cost 0.  The splits of s are the
nonempty subsets p of s without its lowest member, in increasing order, and the first minimum
is kept (a strict < from INF, so a subset whose splits all cost >= INF keeps INF and no split).

Only the costs are computed for every subset: a minimum needs no order (three-operand minima over
all splits, INF included; a NaN split never wins), 1.5 operations per split where carrying the best
split along takes 4 in a serial chain.  A rebuilt treelet asks for the splits of its own few
subsets, which are searched again in order then; the full set's split, always asked for, is
tracked here in two interleaved first-minimum chains over the two halves of its splits (the
second half's minimum is kept only if it is strictly smaller).

Run from this directory:  python gen_treelet_dp.py > treelet_dp_unrolled.cuh
"""
import sys


def subsets_of(mask):
    """Nonempty subsets of mask in increasing numeric order."""
    out = []
    p = mask & -mask
    while p:
        out.append(p)
        p = (p - mask) & mask
    return out


def emit(n, w):
    full = (1 << n) - 1
    w(f"// {n} leaves: {sum(len(subsets_of(s & (s - 1))) for s in range(1, full + 1) if bin(s).count('1') > 1)} "
      f"split evaluations.\n")
    w(f"__device__ __forceinline__ uint32_t dp_unrolled_{n}(float* __restrict__ A) {{\n")
    for s in range(1, full):
        if bin(s).count("1") == 1:
            w(f"  const float c{s} = 0.0f;\n  A[{s} * 32] = 0.0f;\n")
            continue
        terms = [f"__fadd_rn(c{p}, c{s ^ p})" for p in subsets_of(s & (s - 1))]
        # minima of three, level by level: independent until the last
        while len(terms) > 2:
            level = [f"min3f({', '.join(terms[k:k + 3])})" for k in range(0, len(terms) - len(terms) % 3, 3)]
            terms = level + terms[len(terms) - len(terms) % 3:]
        best = f"min3f(kTlInf, {terms[0]}, {terms[1]})" if len(terms) == 2 else f"fminf(kTlInf, {terms[0]})"
        w(f"  const float c{s} = __fadd_rn({best}, A[{s} * 32]);\n  A[{s} * 32] = c{s};\n")
    splits = subsets_of(full & (full - 1))
    h = (len(splits) + 1) // 2
    w("  float b = kTlInf, b2 = kTlInf, v, v2;\n  uint32_t bp = 0u, bp2 = 0u;\n")
    for k in range(h):
        p = splits[k]
        w(f"  v = __fadd_rn(c{p}, c{full ^ p});\n  if (v < b) {{ b = v; bp = {p}u; }}\n")
        if h + k < len(splits):
            q = splits[h + k]
            w(f"  v2 = __fadd_rn(c{q}, c{full ^ q});\n  if (v2 < b2) {{ b2 = v2; bp2 = {q}u; }}\n")
    w("  return b2 < b ? bp2 : bp;\n}\n\n")


def main():
    w = sys.stdout.write
    w("// treelet_dp_unrolled.cuh -- generated by gen_treelet_dp.py; do not edit.\n")
    w("//\n// The LBVH+ subset DP (src/cuda/lbvh_plus_builder.cu:119-165) for N = 4..7 treelet leaves as\n")
    w("// straight-line code: subset costs in registers; this lane's shared-memory column A (stride 32)\n")
    w("// holds the subsets' areas and receives their costs.  Returns the full set's best split, 0 where\n")
    w("// no split is finite.\n")
    w("#pragma once\n\nnamespace bvhgb {\n\n")
    for n in (4, 5, 6, 7):
        emit(n, w)
    w("}  // namespace bvhgb\n")


if __name__ == "__main__":
    main()
