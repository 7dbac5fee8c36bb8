// pv_log.cuh — the natural logarithm of the pair energies, from a table (P. T. P. Tang, "Table-driven
// implementation of the logarithm function in IEEE floating-point arithmetic", ACM TOMS 16 (1990)
// 378-400; the points chosen as in S. Gal and B. Bachelis, "An accurate elementary mathematical library
// for the IEEE floating point standard", ACM TOMS 17 (1991) 26-45).
//
//   v = 2^k m,  m in [0.707, 1.414),  j: the table's point nearest to m,  r = c_j m - 1,  |r| <= 2^-8
//   log v = (k log 2 - log c_j) + r + r^2 p(r)
//
// c_j lies within 2^-16 of 1/(1 + j/128) (2/(1 + j/128) for the points above sqrt 2), where -log c_j is
// a multiple of 2^-42 to 0.01 units of its last place; log 2 is split there as well, so that the sum in
// brackets is exact. The points at 1 have c = 1 and log c = 0, so that the result keeps its relative
// accuracy through the zero at v = 1. p has degree 5 (Chebyshev interpolation, 1e-19 of r). Twelve
// FP64 instructions and no branch, for a normal v > 0; within 1.1 units of the last place. The library's
// logarithm has branches, which keep a loop's pairs from overlapping.
#pragma once

#include <stdint.h>

#if defined(__CUDACC__)
#define PVL_HD __host__ __device__ __forceinline__
#define PVL_TABLE __device__ const
#else
#include <cmath>
#include <cstring>
#define PVL_HD inline
#define PVL_TABLE static const
#endif

namespace pvb {

struct alignas(16) LogPoint {
    double c, t;  // c_j and -log c_j, a multiple of 2^-42
};
constexpr int kLogPoints = 129;

namespace {
PVL_TABLE LogPoint kLogTable[kLogPoints] = {
    {0x1.0000000000000p+0, 0x0.0p+0}, {0x1.fc0652f798ac0p-1, 0x1.fed2d841c0000p-8},
    {0x1.f81e77c5cd2d7p-1, 0x1.fc4e21e880000p-7}, {0x1.f445e56d6f9adp-1, 0x1.7ba096bf10000p-6},
    {0x1.f07dd676cdb73p-1, 0x1.f7f10bb010000p-6}, {0x1.ecc21e558e682p-1, 0x1.39cd435d20000p-5},
    {0x1.e91333712f4c8p-1, 0x1.7743f1bb60000p-5}, {0x1.e574c7dd0b800p-1, 0x1.b41b2a64e8000p-5},
    {0x1.e1e00d4894ad2p-1, 0x1.f0c22a3e58000p-5}, {0x1.de5ec4cbe6fcdp-1, 0x1.1647f9dc68000p-4},
    {0x1.dae60ec9c5c06p-1, 0x1.341d39d574000p-4}, {0x1.d77cf0a6b4aafp-1, 0x1.51a3094dc0000p-4},
    {0x1.d41c012abff76p-1, 0x1.6f181e7c08000p-4}, {0x1.d0ca62631762cp-1, 0x1.8c3cda5c1c000p-4},
    {0x1.cd849afc9c5bdp-1, 0x1.a92df42458000p-4}, {0x1.ca4c3a97f7771p-1, 0x1.c5dbfd4a3c000p-4},
    {0x1.c71cecd185dfep-1, 0x1.e26c238590000p-4}, {0x1.c3f852ef74c85p-1, 0x1.fecea384a4000p-4},
    {0x1.c0dfff4d1cdd7p-1, 0x1.0d79eafd76000p-3}, {0x1.bdd1768a1821cp-1, 0x1.1b7874caae000p-3},
    {0x1.bad1321b50fdep-1, 0x1.294da7c734000p-3}, {0x1.b7d521de54931p-1, 0x1.37275c524c000p-3},
    {0x1.b4e9c8bc0ae43p-1, 0x1.44cad9df22000p-3}, {0x1.b2021f65e40f1p-1, 0x1.52745a138c000p-3},
    {0x1.af27c62b3d1fap-1, 0x1.5ff619bdae000p-3}, {0x1.ac557b0d4cb41p-1, 0x1.6d684a1d5a000p-3},
    {0x1.a98e8a002837cp-1, 0x1.7aba98008e000p-3}, {0x1.a6d17afdcdbe2p-1, 0x1.87f35a9778000p-3},
    {0x1.a41b073a2416ep-1, 0x1.9521e694b8000p-3}, {0x1.a16c507d479b1p-1, 0x1.a2405718d4000p-3},
    {0x1.9eca63916ee57p-1, 0x1.af35494d4c000p-3}, {0x1.9c2e806dfa9bdp-1, 0x1.bc21592380000p-3},
    {0x1.999936482ff7cp-1, 0x1.c9016d10f6000p-3}, {0x1.970fc6a97c53cp-1, 0x1.d5bab733a8000p-3},
    {0x1.948af55e0705ep-1, 0x1.e270fcb6b0000p-3}, {0x1.921001ab5ce55p-1, 0x1.ef09543d0a000p-3},
    {0x1.8f9cfb7ce6074p-1, 0x1.fb8cfdf712000p-3}, {0x1.8d2efe64cdecbp-1, 0x1.040531706d000p-2},
    {0x1.8aca3050034f2p-1, 0x1.0a35e0d949000p-2}, {0x1.886d0e04a04f5p-1, 0x1.105c2f084c000p-2},
    {0x1.8618d6821e41bp-1, 0x1.167497a559000p-2}, {0x1.83c8d2643e585p-1, 0x1.1c8b408642000p-2},
    {0x1.8182f5476830ap-1, 0x1.2290443927000p-2}, {0x1.7f3fb68419f21p-1, 0x1.2897659557000p-2},
    {0x1.7d06409d414b0p-1, 0x1.2e8d5e0787000p-2}, {0x1.7ad32877e4607p-1, 0x1.347b10466b000p-2},
    {0x1.78a48c27f8c45p-1, 0x1.3a656849f5000p-2}, {0x1.767e1d4085382p-1, 0x1.4042306c15000p-2},
    {0x1.745e196f90bccp-1, 0x1.4615f62fee000p-2}, {0x1.7242614bb6a48p-1, 0x1.4be6644218000p-2},
    {0x1.702d7ac9f6d03p-1, 0x1.51ac5af172000p-2}, {0x1.6e1f278adfac7p-1, 0x1.57684edc04000p-2},
    {0x1.6c17f7f74d8acp-1, 0x1.5d18728f6b000p-2}, {0x1.6a152127c981cp+0, -0x1.6303f2766d000p-2},
    {0x1.6816fb990492fp+0, -0x1.5d5d397080000p-2}, {0x1.661e96923531cp+0, -0x1.57beebc694000p-2},
    {0x1.642b715773600p+0, -0x1.5227c64dc2000p-2}, {0x1.62404e29e0be2p+0, -0x1.4c9febd20f000p-2},
    {0x1.605970e2abad4p+0, -0x1.471ccc37ef000p-2}, {0x1.5e75c8d600bfap+0, -0x1.419b690ea8000p-2},
    {0x1.5c989d930be54p+0, -0x1.3c25765323000p-2}, {0x1.5ac1aa0d473a4p+0, -0x1.36ba61992d000p-2},
    {0x1.58ed374c5aef4p+0, -0x1.314f5a47e2000p-2}, {0x1.571f6483b7976p+0, -0x1.2bf0b7c686000p-2},
    {0x1.55544fcb2e4afp+0, -0x1.26931073ac000p-2}, {0x1.5390538e41658p+0, -0x1.214392c9d6000p-2},
    {0x1.51d10e371260dp+0, -0x1.1bfb494c3a000p-2}, {0x1.501611d842f0cp+0, -0x1.16b90b186b000p-2},
    {0x1.4e5f4fc228ee5p+0, -0x1.117ccc6337000p-2}, {0x1.4caa9b493fafap+0, -0x1.0c3ffc728a000p-2},
    {0x1.4afd1a770aaf3p+0, -0x1.07128fe501000p-2}, {0x1.495317996e0a7p+0, -0x1.01e942c329000p-2},
    {0x1.47adbd409c0e2p+0, -0x1.f98fa59ec2000p-3}, {0x1.460ddcb58e58fp+0, -0x1.ef61f09f16000p-3},
    {0x1.4470b2751cb69p+0, -0x1.e538567e4a000p-3}, {0x1.42d7963499edep+0, -0x1.db1b7be756000p-3},
    {0x1.4140506cd7762p+0, -0x1.d0fd7fd9f4000p-3}, {0x1.3fafc3580695cp+0, -0x1.c6fdb7daaa000p-3},
    {0x1.3e22b10271f9fp+0, -0x1.bd07c70374000p-3}, {0x1.3c983df6a8077p+0, -0x1.b316564612000p-3},
    {0x1.3b1356a9a1622p+0, -0x1.a93c8716f2000p-3}, {0x1.399223a619c79p+0, -0x1.9f6eb94500000p-3},
    {0x1.38127b3218f51p+0, -0x1.959ef64562000p-3}, {0x1.3697e410c655ap+0, -0x1.8be4867f8e000p-3},
    {0x1.35209e4342a19p+0, -0x1.82342ececc000p-3}, {0x1.33af7810eea2dp+0, -0x1.78a0cf8102000p-3},
    {0x1.323efbd02d87ep+0, -0x1.6f065cb5d6000p-3}, {0x1.30d25aa3a50fep+0, -0x1.657a3ce27a000p-3},
    {0x1.2f682696c4ae1p+0, -0x1.5bf30b2ee4000p-3}, {0x1.2e016a4f78b5cp+0, -0x1.5277f73276000p-3},
    {0x1.2c9edbcbdee44p+0, -0x1.490e118e04000p-3}, {0x1.2b408ccb5ba68p+0, -0x1.3fb61de91c000p-3},
    {0x1.29e37623aab2ap+0, -0x1.365b973574000p-3}, {0x1.288a15fddc140p+0, -0x1.2d0fb8a71c000p-3},
    {0x1.27354e7c548c3p+0, -0x1.23d8e322f2000p-3}, {0x1.25e21a525fec7p+0, -0x1.1aa25f504a000p-3},
    {0x1.2492d962c6f21p+0, -0x1.117cd9d4f6000p-3}, {0x1.234501b81fc98p+0, -0x1.0856bf7006000p-3},
    {0x1.21fb4382f9575p+0, -0x1.fe862d377c000p-4}, {0x1.20b37ae9af618p+0, -0x1.ec65f7fe3c000p-4},
    {0x1.1f70a28316202p+0, -0x1.da77820374000p-4}, {0x1.1e2e5af3426e1p+0, -0x1.c87cf5d324000p-4},
    {0x1.1cf02f2631447p+0, -0x1.b6a92e9f80000p-4}, {0x1.1bb3cc54282bbp+0, -0x1.a4db3a0580000p-4},
    {0x1.1a7c045696dc4p+0, -0x1.933c24bbe8000p-4}, {0x1.194642af32b3fp+0, -0x1.81a70e0430000p-4},
    {0x1.181076e99602bp+0, -0x1.6ffdfbbfa4000p-4}, {0x1.16dfc8f26e6ddp+0, -0x1.5e8c7c3f90000p-4},
    {0x1.15b1a4b56eb96p+0, -0x1.4d2d5345b8000p-4}, {0x1.1485cad980876p+0, -0x1.3bdd2732b8000p-4},
    {0x1.135cb9f0846d7p+0, -0x1.2aa3981dcc000p-4}, {0x1.123658cd3d718p+0, -0x1.197f8b89d0000p-4},
    {0x1.1111fe35bcdd1p+0, -0x1.08677079ec000p-4}, {0x1.0fee10c8392d2p+0, -0x1.ee86d583a8000p-5},
    {0x1.0ece82aea41d6p+0, -0x1.cc9e2df6f0000p-5}, {0x1.0db187fb77011p+0, -0x1.aadfaf8230000p-5},
    {0x1.0c97f263812e8p+0, -0x1.8965021a00000p-5}, {0x1.0b7d8a1cd2302p+0, -0x1.67adf4d440000p-5},
    {0x1.0a686d469a0bap+0, -0x1.46760d7bf0000p-5}, {0x1.0953c3709a993p+0, -0x1.2529652cf0000p-5},
    {0x1.0842985313cacp+0, -0x1.04264aa9a0000p-5}, {0x1.0732df095c1efp+0, -0x1.c65beac090000p-6},
    {0x1.0624543904582p+0, -0x1.8470e26f60000p-6}, {0x1.051910cb4f8c6p+0, -0x1.430f702980000p-6},
    {0x1.040fca12d37e4p+0, -0x1.01e8202490000p-6}, {0x1.03081e9e03c8cp+0, -0x1.81c7ab1080000p-7},
    {0x1.0204ed1a650b8p+0, -0x1.0172f73e40000p-7}, {0x1.0101925c83acfp+0, -0x1.01111f93c0000p-8},
    {0x1.0000000000000p+0, 0x0.0p+0},
};
} // namespace

PVL_HD double log_words(uint32_t hi, uint32_t lo) {
#if defined(__CUDA_ARCH__)
    return __hiloint2double(static_cast<int>(hi), static_cast<int>(lo));
#else
    const uint64_t b = static_cast<uint64_t>(hi) << 32 | lo;
    double v;
    __builtin_memcpy(&v, &b, sizeof v);
    return v;
#endif
}
PVL_HD uint32_t log_high(double v) {
#if defined(__CUDA_ARCH__)
    return static_cast<uint32_t>(__double2hiint(v));
#else
    uint64_t b;
    __builtin_memcpy(&b, &v, sizeof b);
    return static_cast<uint32_t>(b >> 32);
#endif
}
PVL_HD uint32_t log_low(double v) {
#if defined(__CUDA_ARCH__)
    return static_cast<uint32_t>(__double2loint(v));
#else
    uint64_t b;
    __builtin_memcpy(&b, &v, sizeof b);
    return static_cast<uint32_t>(b);
#endif
}

// Whether log_normal() serves v: positive, normal, finite.
PVL_HD bool log_is_normal(double v) { return log_high(v) - 0x00100000u < 0x7fe00000u; }

PVL_HD double log_normal(double v, const LogPoint *table) {
    const uint32_t hi = log_high(v);
    const uint32_t j = ((hi & 0xfffffu) + (1u << 12)) >> 13;  // 0 .. 128
    const uint32_t biased = (hi >> 20) + (j >= 53 ? 1 : 0);   // k + 1023
    const double m = log_words(hi - ((biased - 1023u) << 20), log_low(v));
    const LogPoint p = table[j];
    // k without a conversion: 2^52 + biased, less 2^52 + 1023
    const double k = log_words(0x43300000u, biased) - 4503599627371519.0;
    const double lead = fma(k, 0x1.62e42fefa3800p-1, p.t);  // exact
    const double r = fma(m, p.c, -1.0);
    const double r2 = r * r;
    const double p0 = fma(r, 0x1.5555555555556p-2, -0.5);
    const double p1 = fma(r, 0x1.999999991918dp-3, -0x1.ffffffff6f6f2p-3);
    const double p2 = fma(r, 0x1.24939f25e308cp-3, -0x1.5556d616c84a3p-3);
    const double tail = fma(k, 0x1.ef35793c76730p-45, r);
    return lead + fma(r2, fma(r2, fma(r2, p2, p1), p0), tail);
}

} // namespace pvb
