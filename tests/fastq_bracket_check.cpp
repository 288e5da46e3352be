// CPU check of the float reconstruction that the common path runs
// (dequant_f32_bracket, faz_gb300/csrc/fastq.cuh) and of the quantiser around it, at
// what fastq_check.cpp gives to their predecessors: values of the whole float range
// (denormals, infinities and NaN among them), sums on and beside the midpoints of two
// floats, cancellation, powers of two, signed zeros, halves up to the largest radius
// (65536), bounds over the fast path's whole range (2^-60 to 2^60).  A decided result
// equals the double computation's bit for bit.  (How many
// stay undecided is printed and not judged: sums of two floats fall on midpoints
// exactly, and often.)
// Usage: fastq_bracket_check <cases> <seed>; prints counts; exit 1 on any mismatch.
#include <cinttypes>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../faz_gb300/csrc/fastq.cuh"

using namespace faz;

static float any_float(std::mt19937_64 &rng) { return f32_from_bits((uint32_t)rng()); }

static bool same(float a, float b) { return f32_bits(a) == f32_bits(b); }

int main(int argc, char **argv) {
    const uint64_t cases = argc > 1 ? strtoull(argv[1], 0, 10) : 1000000;
    std::mt19937_64 rng(argc > 2 ? strtoull(argv[2], 0, 10) : 1);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    uint64_t decided = 0, undecided = 0, bad = 0, q_decided = 0, q_bad = 0;
    for (uint64_t i = 0; i < cases; i++) {
        double eb;
        switch (rng() % 4) {
        case 0: eb = std::ldexp(1.0 + U(rng), (int)(rng() % 120) - 60); break;
        case 1: eb = std::ldexp(1.0, (int)(rng() % 121) - 60); break;
        case 2: eb = (double)(1 + rng() % 1000) * std::pow(10.0, -(int)(rng() % 9)); break;
        default: eb = 1e-3 * (double)(float)(130 * U(rng) + 1e-9);
        }
        if (!(eb >= 0x1p-60 && eb <= 0x1p60)) eb = 1e-3;
        const float eh = (float)eb, el = (float)(eb - (double)eh);
        // ---- reconstruction
        int half = (int)(rng() % 131073) - 65536;
        if (rng() % 4 == 0) half = (int)(rng() % 9) - 4;
        const double step = (double)(2 * half) * eb;
        float pred;
        const int pk = (int)(rng() % 8);
        switch (pk) {
        case 0: pred = (float)((U(rng) - 0.5) * 200 * eb); break;
        case 1: {  // a sum beside the midpoint of two floats
            const float v = (float)((U(rng) - 0.5) * std::ldexp(eb, (int)(rng() % 40)));
            double mid = (double)v + 0.5 * (double)(std::nextafter(v, INFINITY) - v);
            mid += (U(rng) - 0.5) * std::ldexp(std::fabs((double)v), -(int)(30 + rng() % 30));
            pred = (float)(mid - step);
            break;
        }
        case 2: pred = (float)(-step * (1 + (U(rng) - 0.5) * 1e-6)); break;  // cancellation
        case 3: pred = std::nextafter((float)-step, rng() & 1 ? INFINITY : -INFINITY); break;
        case 4: pred = std::ldexp(rng() & 1 ? 1.0f : -1.0f, (int)(rng() % 276) - 149); break;
        case 5: pred = rng() & 1 ? 0.0f : -0.0f; break;
        case 6: pred = f32_from_bits((uint32_t)rng() & 0x807fffffu); break;  // denormal
        default: pred = any_float(rng);
        }
        float out;
        const bool und = dequant_f32_bracket(pred, (float)half, 2.0f * eh, 2.0f * el, out);
        const float ref = (float)((double)pred + step);
        undecided += und;
        decided += !und;
        if (!und && !same(out, ref)) {
            if (bad++ < 10)
                std::printf("bracket: pred=%a half=%d eb=%a got=%a want=%a\n", (double)pred, half, eb, (double)out,
                            (double)ref);
        }
        // ---- quantiser: what is decided is what the double computation gives
        int radius = 65536 >> (rng() % 17);
        float orig;
        switch (rng() % 5) {
        case 0: orig = any_float(rng); break;
        case 1: orig = (float)((double)pred + (2.0 * (int)(rng() % 70000) - 69999 + (U(rng) - 0.5) * 1e-6) * eb); break;
        case 2: orig = (float)((double)pred + step); break;
        case 3: orig = std::nextafter(pred, rng() & 1 ? INFINITY : -INFINITY); break;
        default: orig = pred + (float)((U(rng) - 0.5) * 10 * eb);
        }
        const double recip = 1.0 / eb;
        const float rh = (float)recip, rl = (float)(recip - (double)rh);
        float eblo = (float)eb;
        if ((double)eblo > eb) eblo = std::nextafter(eblo, 0.0f);
        float q_out, want = orig;
        bool q_und;
        const int code = quantize_f32_straight(orig, pred, rh, rl, eh, el, eblo, (float)(2 * radius), radius, q_out, q_und);
        int want_code = 0;
        const float diff = orig - pred;
        const double x = (double)std::fabs(diff) * recip;
        if (x < 2147483647.0 && (int)x + 1 < 2 * radius) {
            const int h = ((int)x + 1) >> 1, q2 = diff < 0 ? -(h << 1) : h << 1;
            const float dec = (float)((double)pred + (double)q2 * eb), err = dec - orig;
            if (!(std::fabs((double)err) > eb)) {
                want = dec;
                want_code = diff < 0 ? radius - h : radius + h;
            }
        }
        if (q_und) continue;
        q_decided++;
        if (code != want_code || !same(q_out, want)) {
            if (q_bad++ < 10)
                std::printf("quantiser: orig=%a pred=%a eb=%a radius=%d got=(%d,%a) want=(%d,%a)\n", (double)orig,
                            (double)pred, eb, radius, code, (double)q_out, want_code, (double)want);
        }
    }
    std::printf("decided=%" PRIu64 " undecided=%" PRIu64 " bad=%" PRIu64 " quantised=%" PRIu64 " bad=%" PRIu64 "\n",
                decided, undecided, bad, q_decided, q_bad);
    return bad || q_bad;
}
