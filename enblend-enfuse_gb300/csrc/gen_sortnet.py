"""Generate enb_sortnet.cuh: Batcher's odd-even merge sorting networks for the
local-entropy windows (3x3 = 9 and 5x5 = 25 keys), padded to 16 and 32 keys
and pruned of every comparator that touches a padding position (padding keys
are the maximum key, so such comparators never exchange); and his odd-even
merges of two sorted lists, from which the windows of vertically adjacent
pixels are sorted with their common rows sorted once.

Usage: python gen_sortnet.py > enb_sortnet.cuh
"""


def batcher(n_pow2: int, live: int):
    pairs = []
    p = 1
    while p < n_pow2:
        k = p
        while k >= 1:
            j = k % p
            while j + k < n_pow2:
                for i in range(k):
                    a, b = i + j, i + j + k
                    if a // (2 * p) == b // (2 * p) and b < live:
                        pairs.append((a, b))
                j += 2 * k
            k //= 2
        p *= 2
    return pairs


def check(pairs, live):
    import itertools
    import random
    rnd = random.Random(1)
    for _ in range(20000):
        v = [rnd.randrange(6) for _ in range(live)]
        for a, b in pairs:
            if v[a] > v[b]:
                v[a], v[b] = v[b], v[a]
        assert v == sorted(v)


def merge(a, b, pairs):
    """Odd-even merge of the sorted wire lists a and b (Batcher 1968; Knuth
    5.3.4 for any lengths): appends its comparators to pairs, returns the
    wires in ascending order of their keys."""
    if not a or not b:
        return a + b
    if len(a) == 1 and len(b) == 1:
        pairs.append((a[0], b[0]))
        return [a[0], b[0]]
    v, w = merge(a[0::2], b[0::2], pairs), merge(a[1::2], b[1::2], pairs)
    out = [v[0]]
    for i in range(max(len(w), len(v) - 1)):
        if i < len(w) and i + 1 < len(v):
            pairs.append((w[i], v[i + 1]))
        out += w[i:i + 1] + v[i + 1:i + 2]
    return out


def check_merge(m, n, pairs, out):
    # the 0-1 principle: every pair of sorted 0-1 lists
    for i in range(m + 1):
        for j in range(n + 1):
            v = [0] * i + [1] * (m - i) + [0] * j + [1] * (n - j)
            for a, b in pairs:
                if v[a] > v[b]:
                    v[a], v[b] = v[b], v[a]
            r = [v[x] for x in out]
            assert r == sorted(r)


SORT = {3: [(0, 1), (1, 2), (0, 1)],
        5: [(0, 1), (3, 4), (2, 4), (2, 3), (0, 3), (0, 2), (1, 4), (1, 3), (1, 2)]}


def main():
    print("// enb_sortnet.cuh -- generated by gen_sortnet.py (Batcher's odd-even merge")
    print("// sort, pruned to the live keys); do not edit by hand.")
    print("#pragma once")
    print()
    print("#include <stdint.h>")
    print()
    print("namespace enb {")
    print()
    print("// Compare-exchange of two 32-bit keys (ascending).")
    print("struct CeU32 {")
    print("    __device__ __forceinline__ void operator()(uint32_t& a, uint32_t& b) const")
    print("    {")
    print("        const uint32_t lo = min(a, b);")
    print("        b = max(a, b);")
    print("        a = lo;")
    print("    }")
    print("};")
    print()
    print("// Compare-exchange of the two 16-bit halves of two words independently")
    print("// (two windows sorted at once, one per half).")
    print("struct CeU16x2 {")
    print("    __device__ __forceinline__ void operator()(uint32_t& a, uint32_t& b) const")
    print("    {")
    print("        uint32_t lo, hi;")
    print('        asm("min.u16x2 %0, %1, %2;" : "=r"(lo) : "r"(a), "r"(b));')
    print('        asm("max.u16x2 %0, %1, %2;" : "=r"(hi) : "r"(a), "r"(b));')
    print("        a = lo;")
    print("        b = hi;")
    print("    }")
    print("};")
    for live, n in ((9, 16), (25, 32)):
        pairs = batcher(n, live)
        check(pairs, live)
        print()
        print(f"// Sorts k[0..{live - 1}] ascending ({len(pairs)} comparators).")
        print("template <class CE = CeU32>")
        print(f"__device__ __forceinline__ void sortnet{live}(uint32_t (&k)[{live}], CE ce = CE())")
        print("{")
        for a, b in pairs:
            print(f"    ce(k[{a}], k[{b}]);")
        print("}")
    for n in (3, 5):
        check(SORT[n], n)
        print()
        print(f"// Sorts k[0..{n - 1}] ascending ({len(SORT[n])} comparators).")
        print("template <class CE = CeU32>")
        print(f"__device__ __forceinline__ void sort_row(uint32_t (&k)[{n}], CE ce = CE())")
        print("{")
        for a, b in SORT[n]:
            print(f"    ce(k[{a}], k[{b}]);")
        print("}")
    for m, n in ((3, 3), (3, 6), (5, 5), (10, 10), (5, 20)):
        pairs = []
        out = merge(list(range(m)), list(range(m, m + n)), pairs)
        check_merge(m, n, pairs, out)
        print()
        print(f"// Merges the sorted lists a and b into o ({len(pairs)} comparators).")
        print("template <class CE = CeU32>")
        print(f"__device__ __forceinline__ void merge_sorted(const uint32_t (&a)[{m}], const uint32_t (&b)[{n}], "
              f"uint32_t (&o)[{m + n}], CE ce = CE())")
        print("{")
        print(f"    uint32_t k[{m + n}];")
        print("#pragma unroll")
        print(f"    for (int i = 0; i < {m}; ++i) {{")
        print("        k[i] = a[i];")
        print("    }")
        print("#pragma unroll")
        print(f"    for (int i = 0; i < {n}; ++i) {{")
        print(f"        k[{m} + i] = b[i];")
        print("    }")
        for x, y in pairs:
            print(f"    ce(k[{x}], k[{y}]);")
        for i, x in enumerate(out):
            print(f"    o[{i}] = k[{x}];")
        print("}")
    print()
    print("}  // namespace enb")


if __name__ == "__main__":
    main()
