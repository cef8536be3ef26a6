// enb_sortnet.cuh -- generated by gen_sortnet.py (Batcher's odd-even merge
// sort, pruned to the live keys); do not edit by hand.
#pragma once

#include <stdint.h>

namespace enb {

// Compare-exchange of two 32-bit keys (ascending).
struct CeU32 {
    __device__ __forceinline__ void operator()(uint32_t& a, uint32_t& b) const
    {
        const uint32_t lo = min(a, b);
        b = max(a, b);
        a = lo;
    }
};

// Compare-exchange of the two 16-bit halves of two words independently
// (two windows sorted at once, one per half).
struct CeU16x2 {
    __device__ __forceinline__ void operator()(uint32_t& a, uint32_t& b) const
    {
        uint32_t lo, hi;
        asm("min.u16x2 %0, %1, %2;" : "=r"(lo) : "r"(a), "r"(b));
        asm("max.u16x2 %0, %1, %2;" : "=r"(hi) : "r"(a), "r"(b));
        a = lo;
        b = hi;
    }
};

// Sorts k[0..8] ascending (28 comparators).
template <class CE = CeU32>
__device__ __forceinline__ void sortnet9(uint32_t (&k)[9], CE ce = CE())
{
    ce(k[0], k[1]);
    ce(k[2], k[3]);
    ce(k[4], k[5]);
    ce(k[6], k[7]);
    ce(k[0], k[2]);
    ce(k[1], k[3]);
    ce(k[4], k[6]);
    ce(k[5], k[7]);
    ce(k[1], k[2]);
    ce(k[5], k[6]);
    ce(k[0], k[4]);
    ce(k[1], k[5]);
    ce(k[2], k[6]);
    ce(k[3], k[7]);
    ce(k[2], k[4]);
    ce(k[3], k[5]);
    ce(k[1], k[2]);
    ce(k[3], k[4]);
    ce(k[5], k[6]);
    ce(k[0], k[8]);
    ce(k[4], k[8]);
    ce(k[2], k[4]);
    ce(k[3], k[5]);
    ce(k[6], k[8]);
    ce(k[1], k[2]);
    ce(k[3], k[4]);
    ce(k[5], k[6]);
    ce(k[7], k[8]);
}

// Sorts k[0..24] ascending (140 comparators).
template <class CE = CeU32>
__device__ __forceinline__ void sortnet25(uint32_t (&k)[25], CE ce = CE())
{
    ce(k[0], k[1]);
    ce(k[2], k[3]);
    ce(k[4], k[5]);
    ce(k[6], k[7]);
    ce(k[8], k[9]);
    ce(k[10], k[11]);
    ce(k[12], k[13]);
    ce(k[14], k[15]);
    ce(k[16], k[17]);
    ce(k[18], k[19]);
    ce(k[20], k[21]);
    ce(k[22], k[23]);
    ce(k[0], k[2]);
    ce(k[1], k[3]);
    ce(k[4], k[6]);
    ce(k[5], k[7]);
    ce(k[8], k[10]);
    ce(k[9], k[11]);
    ce(k[12], k[14]);
    ce(k[13], k[15]);
    ce(k[16], k[18]);
    ce(k[17], k[19]);
    ce(k[20], k[22]);
    ce(k[21], k[23]);
    ce(k[1], k[2]);
    ce(k[5], k[6]);
    ce(k[9], k[10]);
    ce(k[13], k[14]);
    ce(k[17], k[18]);
    ce(k[21], k[22]);
    ce(k[0], k[4]);
    ce(k[1], k[5]);
    ce(k[2], k[6]);
    ce(k[3], k[7]);
    ce(k[8], k[12]);
    ce(k[9], k[13]);
    ce(k[10], k[14]);
    ce(k[11], k[15]);
    ce(k[16], k[20]);
    ce(k[17], k[21]);
    ce(k[18], k[22]);
    ce(k[19], k[23]);
    ce(k[2], k[4]);
    ce(k[3], k[5]);
    ce(k[10], k[12]);
    ce(k[11], k[13]);
    ce(k[18], k[20]);
    ce(k[19], k[21]);
    ce(k[1], k[2]);
    ce(k[3], k[4]);
    ce(k[5], k[6]);
    ce(k[9], k[10]);
    ce(k[11], k[12]);
    ce(k[13], k[14]);
    ce(k[17], k[18]);
    ce(k[19], k[20]);
    ce(k[21], k[22]);
    ce(k[0], k[8]);
    ce(k[1], k[9]);
    ce(k[2], k[10]);
    ce(k[3], k[11]);
    ce(k[4], k[12]);
    ce(k[5], k[13]);
    ce(k[6], k[14]);
    ce(k[7], k[15]);
    ce(k[16], k[24]);
    ce(k[4], k[8]);
    ce(k[5], k[9]);
    ce(k[6], k[10]);
    ce(k[7], k[11]);
    ce(k[20], k[24]);
    ce(k[2], k[4]);
    ce(k[3], k[5]);
    ce(k[6], k[8]);
    ce(k[7], k[9]);
    ce(k[10], k[12]);
    ce(k[11], k[13]);
    ce(k[18], k[20]);
    ce(k[19], k[21]);
    ce(k[22], k[24]);
    ce(k[1], k[2]);
    ce(k[3], k[4]);
    ce(k[5], k[6]);
    ce(k[7], k[8]);
    ce(k[9], k[10]);
    ce(k[11], k[12]);
    ce(k[13], k[14]);
    ce(k[17], k[18]);
    ce(k[19], k[20]);
    ce(k[21], k[22]);
    ce(k[23], k[24]);
    ce(k[0], k[16]);
    ce(k[1], k[17]);
    ce(k[2], k[18]);
    ce(k[3], k[19]);
    ce(k[4], k[20]);
    ce(k[5], k[21]);
    ce(k[6], k[22]);
    ce(k[7], k[23]);
    ce(k[8], k[24]);
    ce(k[8], k[16]);
    ce(k[9], k[17]);
    ce(k[10], k[18]);
    ce(k[11], k[19]);
    ce(k[12], k[20]);
    ce(k[13], k[21]);
    ce(k[14], k[22]);
    ce(k[15], k[23]);
    ce(k[4], k[8]);
    ce(k[5], k[9]);
    ce(k[6], k[10]);
    ce(k[7], k[11]);
    ce(k[12], k[16]);
    ce(k[13], k[17]);
    ce(k[14], k[18]);
    ce(k[15], k[19]);
    ce(k[20], k[24]);
    ce(k[2], k[4]);
    ce(k[3], k[5]);
    ce(k[6], k[8]);
    ce(k[7], k[9]);
    ce(k[10], k[12]);
    ce(k[11], k[13]);
    ce(k[14], k[16]);
    ce(k[15], k[17]);
    ce(k[18], k[20]);
    ce(k[19], k[21]);
    ce(k[22], k[24]);
    ce(k[1], k[2]);
    ce(k[3], k[4]);
    ce(k[5], k[6]);
    ce(k[7], k[8]);
    ce(k[9], k[10]);
    ce(k[11], k[12]);
    ce(k[13], k[14]);
    ce(k[15], k[16]);
    ce(k[17], k[18]);
    ce(k[19], k[20]);
    ce(k[21], k[22]);
    ce(k[23], k[24]);
}

// Sorts k[0..2] ascending (3 comparators).
template <class CE = CeU32>
__device__ __forceinline__ void sort_row(uint32_t (&k)[3], CE ce = CE())
{
    ce(k[0], k[1]);
    ce(k[1], k[2]);
    ce(k[0], k[1]);
}

// Sorts k[0..4] ascending (9 comparators).
template <class CE = CeU32>
__device__ __forceinline__ void sort_row(uint32_t (&k)[5], CE ce = CE())
{
    ce(k[0], k[1]);
    ce(k[3], k[4]);
    ce(k[2], k[4]);
    ce(k[2], k[3]);
    ce(k[0], k[3]);
    ce(k[0], k[2]);
    ce(k[1], k[4]);
    ce(k[1], k[3]);
    ce(k[1], k[2]);
}

// Merges the sorted lists a and b into o (6 comparators).
template <class CE = CeU32>
__device__ __forceinline__ void merge_sorted(const uint32_t (&a)[3], const uint32_t (&b)[3], uint32_t (&o)[6], CE ce = CE())
{
    uint32_t k[6];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        k[i] = a[i];
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        k[3 + i] = b[i];
    }
    ce(k[0], k[3]);
    ce(k[2], k[5]);
    ce(k[2], k[3]);
    ce(k[1], k[4]);
    ce(k[1], k[2]);
    ce(k[4], k[3]);
    o[0] = k[0];
    o[1] = k[1];
    o[2] = k[2];
    o[3] = k[4];
    o[4] = k[3];
    o[5] = k[5];
}

// Merges the sorted lists a and b into o (12 comparators).
template <class CE = CeU32>
__device__ __forceinline__ void merge_sorted(const uint32_t (&a)[3], const uint32_t (&b)[6], uint32_t (&o)[9], CE ce = CE())
{
    uint32_t k[9];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        k[i] = a[i];
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        k[3 + i] = b[i];
    }
    ce(k[0], k[3]);
    ce(k[7], k[3]);
    ce(k[2], k[5]);
    ce(k[2], k[7]);
    ce(k[5], k[3]);
    ce(k[1], k[4]);
    ce(k[8], k[4]);
    ce(k[6], k[8]);
    ce(k[1], k[2]);
    ce(k[6], k[7]);
    ce(k[8], k[5]);
    ce(k[4], k[3]);
    o[0] = k[0];
    o[1] = k[1];
    o[2] = k[2];
    o[3] = k[6];
    o[4] = k[7];
    o[5] = k[8];
    o[6] = k[5];
    o[7] = k[4];
    o[8] = k[3];
}

// Merges the sorted lists a and b into o (13 comparators).
template <class CE = CeU32>
__device__ __forceinline__ void merge_sorted(const uint32_t (&a)[5], const uint32_t (&b)[5], uint32_t (&o)[10], CE ce = CE())
{
    uint32_t k[10];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        k[i] = a[i];
    }
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        k[5 + i] = b[i];
    }
    ce(k[0], k[5]);
    ce(k[4], k[9]);
    ce(k[4], k[5]);
    ce(k[2], k[7]);
    ce(k[2], k[4]);
    ce(k[7], k[5]);
    ce(k[1], k[6]);
    ce(k[3], k[8]);
    ce(k[3], k[6]);
    ce(k[1], k[2]);
    ce(k[3], k[4]);
    ce(k[6], k[7]);
    ce(k[8], k[5]);
    o[0] = k[0];
    o[1] = k[1];
    o[2] = k[2];
    o[3] = k[3];
    o[4] = k[4];
    o[5] = k[6];
    o[6] = k[7];
    o[7] = k[8];
    o[8] = k[5];
    o[9] = k[9];
}

// Merges the sorted lists a and b into o (35 comparators).
template <class CE = CeU32>
__device__ __forceinline__ void merge_sorted(const uint32_t (&a)[10], const uint32_t (&b)[10], uint32_t (&o)[20], CE ce = CE())
{
    uint32_t k[20];
#pragma unroll
    for (int i = 0; i < 10; ++i) {
        k[i] = a[i];
    }
#pragma unroll
    for (int i = 0; i < 10; ++i) {
        k[10 + i] = b[i];
    }
    ce(k[0], k[10]);
    ce(k[8], k[18]);
    ce(k[8], k[10]);
    ce(k[4], k[14]);
    ce(k[4], k[8]);
    ce(k[14], k[10]);
    ce(k[2], k[12]);
    ce(k[6], k[16]);
    ce(k[6], k[12]);
    ce(k[2], k[4]);
    ce(k[6], k[8]);
    ce(k[12], k[14]);
    ce(k[16], k[10]);
    ce(k[1], k[11]);
    ce(k[9], k[19]);
    ce(k[9], k[11]);
    ce(k[5], k[15]);
    ce(k[5], k[9]);
    ce(k[15], k[11]);
    ce(k[3], k[13]);
    ce(k[7], k[17]);
    ce(k[7], k[13]);
    ce(k[3], k[5]);
    ce(k[7], k[9]);
    ce(k[13], k[15]);
    ce(k[17], k[11]);
    ce(k[1], k[2]);
    ce(k[3], k[4]);
    ce(k[5], k[6]);
    ce(k[7], k[8]);
    ce(k[9], k[12]);
    ce(k[13], k[14]);
    ce(k[15], k[16]);
    ce(k[17], k[10]);
    ce(k[11], k[18]);
    o[0] = k[0];
    o[1] = k[1];
    o[2] = k[2];
    o[3] = k[3];
    o[4] = k[4];
    o[5] = k[5];
    o[6] = k[6];
    o[7] = k[7];
    o[8] = k[8];
    o[9] = k[9];
    o[10] = k[12];
    o[11] = k[13];
    o[12] = k[14];
    o[13] = k[15];
    o[14] = k[16];
    o[15] = k[17];
    o[16] = k[10];
    o[17] = k[11];
    o[18] = k[18];
    o[19] = k[19];
}

// Merges the sorted lists a and b into o (46 comparators).
template <class CE = CeU32>
__device__ __forceinline__ void merge_sorted(const uint32_t (&a)[5], const uint32_t (&b)[20], uint32_t (&o)[25], CE ce = CE())
{
    uint32_t k[25];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        k[i] = a[i];
    }
#pragma unroll
    for (int i = 0; i < 20; ++i) {
        k[5 + i] = b[i];
    }
    ce(k[0], k[5]);
    ce(k[21], k[5]);
    ce(k[13], k[21]);
    ce(k[4], k[9]);
    ce(k[17], k[9]);
    ce(k[4], k[13]);
    ce(k[17], k[21]);
    ce(k[9], k[5]);
    ce(k[2], k[7]);
    ce(k[23], k[7]);
    ce(k[15], k[23]);
    ce(k[11], k[15]);
    ce(k[19], k[23]);
    ce(k[2], k[4]);
    ce(k[11], k[13]);
    ce(k[15], k[17]);
    ce(k[19], k[21]);
    ce(k[23], k[9]);
    ce(k[7], k[5]);
    ce(k[1], k[6]);
    ce(k[22], k[6]);
    ce(k[14], k[22]);
    ce(k[10], k[14]);
    ce(k[18], k[22]);
    ce(k[3], k[8]);
    ce(k[24], k[8]);
    ce(k[16], k[24]);
    ce(k[12], k[16]);
    ce(k[20], k[24]);
    ce(k[3], k[10]);
    ce(k[12], k[14]);
    ce(k[16], k[18]);
    ce(k[20], k[22]);
    ce(k[24], k[6]);
    ce(k[1], k[2]);
    ce(k[3], k[4]);
    ce(k[10], k[11]);
    ce(k[12], k[13]);
    ce(k[14], k[15]);
    ce(k[16], k[17]);
    ce(k[18], k[19]);
    ce(k[20], k[21]);
    ce(k[22], k[23]);
    ce(k[24], k[9]);
    ce(k[6], k[7]);
    ce(k[8], k[5]);
    o[0] = k[0];
    o[1] = k[1];
    o[2] = k[2];
    o[3] = k[3];
    o[4] = k[4];
    o[5] = k[10];
    o[6] = k[11];
    o[7] = k[12];
    o[8] = k[13];
    o[9] = k[14];
    o[10] = k[15];
    o[11] = k[16];
    o[12] = k[17];
    o[13] = k[18];
    o[14] = k[19];
    o[15] = k[20];
    o[16] = k[21];
    o[17] = k[22];
    o[18] = k[23];
    o[19] = k[24];
    o[20] = k[9];
    o[21] = k[6];
    o[22] = k[7];
    o[23] = k[8];
    o[24] = k[5];
}

}  // namespace enb
