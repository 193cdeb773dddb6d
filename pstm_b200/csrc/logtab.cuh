// logtab.cuh -- natural logarithm in FP64 for the curved-ray traveltime.
//
// Table-driven, after P. T. P. Tang, "Table-driven implementation of the
// logarithm function in IEEE floating-point arithmetic", ACM TOMS 16(4), 1990:
// x = 2^e m, m in [1, 2); the top kLogBits bits of m's fraction pick c ~ 1/m, a
// float, and -log c from a table; z = c m - 1, |z| <= 2^-8, and log x = e log 2 -
// log c + log1p(z), with the Taylor polynomial of log1p through z^6.  The next term is
// below 2^-58, so what is left is rounding: the table entry's and those of sums of
// size |log x|, below 2^-53 (0.75 + 3.5 |log x|) together for every positive normal x
// (tests/test_log_table.py).
//
// Why not log(): it is correct nearly to the last bit for any argument, at some
// three times the FP64 instructions.  A curved leg's sample index needs 2^-35, and
// the square roots in the argument are good to 2^-44.  64 entries and the same
// polynomial (2^-50) took the same time.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define PSTM_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#include <cstring>
#define PSTM_HD inline
#endif

namespace pstm {

constexpr int kLogBits = 7;
constexpr int kLogEntries = 1 << kLogBits;
struct alignas(16) LogEntry {
    double c, l;   // 1/m at the middle of the entry's interval, -log c
};

PSTM_HD LogEntry log_entry(int i) {
    const double c = (double)(float)(1.0 / (1.0 + (i + 0.5) / kLogEntries));
    return {c, -log(c)};
}

// log x for x positive, finite and normal.
PSTM_HD double log_by_table(const LogEntry *tab, double x) {
#if defined(__CUDA_ARCH__)
    const uint32_t hi = (uint32_t)__double2hiint(x);
    const double m = __hiloint2double((int)((hi & 0xFFFFFu) | 0x3FF00000u), __double2loint(x));
    // the exponent field in the low word of 2^52, taken off again with the bias
    const double e = __hiloint2double(0x43300000, (int)(hi >> 20)) - (4503599627370496.0 + 1023.0);
#else
    uint64_t u, v;
    std::memcpy(&u, &x, 8);
    const uint32_t hi = (uint32_t)(u >> 32);
    v = (u & 0xFFFFFFFFFFFFFull) | 0x3FF0000000000000ull;
    double m;
    std::memcpy(&m, &v, 8);
    const double e = (double)(int)(hi >> 20) - 1023.0;
#endif
    const LogEntry t = tab[(hi >> (20 - kLogBits)) & (kLogEntries - 1)];
    const double z = fma(t.c, m, -1.0);
    double p = fma(z, -1.0 / 6.0, 1.0 / 5.0);
    p = fma(p, z, -1.0 / 4.0);
    p = fma(p, z, 1.0 / 3.0);
    p = fma(p, z, -1.0 / 2.0);
    return fma(z * z, p, fma(e, 0.69314718055994530942, t.l) + z);
}

}  // namespace pstm
