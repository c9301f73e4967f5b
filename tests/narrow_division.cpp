// Checks meshing.jl_gb300/csrc/mesh_quot.h against the IEEE division: random and
// edge operands of every form, with reciprocal seeds off by up to two ulps either
// way (the device's estimate is good to one).  Prints the number of mismatches.
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

static int g_off = 0;
static float seed(float x) {
    float r = 1.0f / x;
    for (int k = 0; k < abs(g_off); k++) r = nextafterf(r, g_off > 0 ? 2.0f : 0.0f);
    return r;
}
#define MESH_QUOT_SEED(x) seed(x)
#include "mesh_quot.h"

static uint64_t s = 88172645463325252ull;
static uint64_t rnd() {
    s ^= s << 13;
    s ^= s >> 7;
    s ^= s << 17;
    return s;
}
template <class A, class B> static B pun(A a) {
    B b;
    memcpy(&b, &a, sizeof b);
    return b;
}

int main(int argc, char **argv) {
    const long n = argc > 1 ? atol(argv[1]) : 1000000;
    long bad = 0, taken = 0;
    auto check = [&](bool ok, const uint64_t &got, double want) {
        if (!ok) return;
        taken++;
        const uint64_t w = pun<double, uint64_t>(want);
        const unsigned e = (unsigned)(w >> 52) & 0x7ffu;
        bad += e == 0 || e == 0x7ff || w != got;
    };
    for (long i = 0; i < n; i++) {
        g_off = (int)(i % 5) - 2;
        uint64_t a = rnd(), q = 0;
        unsigned f = (unsigned)rnd(), g = (unsigned)(rnd() >> 7);
        switch (i % 7) {  // edges: short and full significands, near powers of two, equal operands
        case 1: a &= ~0ull << (rnd() % 52); f &= ~0u << (rnd() % 23); break;
        case 2: a |= ((1ull << (rnd() % 53)) - 1); f |= (1u << (rnd() % 24)) - 1; break;
        case 3: f = (f & 0xff800000u) | (unsigned)(rnd() % 4); break;
        case 4: f |= 0x7fffffu & ~(unsigned)(rnd() % 4); break;
        case 5: g = f; break;
        case 6: a = pun<double, uint64_t>((double)pun<unsigned, float>(g)); break;
        }
        const double da = pun<uint64_t, double>(a);
        const float df = pun<unsigned, float>(f), dg = pun<unsigned, float>(g);
        check(mesh::quot_f64_f32(a, f, q), q, da / (double)df);
        check(mesh::quot_f32_f32(g, f, q), q, (double)dg / (double)df);
        const int ia = (int)(rnd() >> (rnd() % 64)), id = (int)((long long)rnd() >> (32 + rnd() % 32));
        check(mesh::quot_i32_i32(ia, id, q), q, (double)ia / (double)id);
        check(mesh::quot_f64_i32(a, id, q), q, da / (double)id);
    }
    printf("%ld %ld\n", bad, taken);
    return bad != 0;
}
