// The run forms of the RFI scans (KadanePair32, KadaneBest) over floats as
// the scans meet them, against the full KadaneState: zeros of both signs,
// subnormals, equal values that cancel to exact zeros, infinities, NaN, and
// channels that are left out (KadaneBest is given 0 for them, the full state
// nothing). Prints "bad N" with N the mismatches.

#include <cmath>
#include <cstdio>
#include <limits>
#include <random>

#include "rfi_types.hpp"

using namespace fb::rfi;

namespace {

bool same(double a, double b) { return (std::isnan(a) && std::isnan(b)) || a == b; }
bool same(const Run& a, const Run& b) { return same(a.sum, b.sum) && a.start == b.start && a.end == b.end; }
bool same(const KadaneState& a, const KadaneState& b) {
    return same(a.total, b.total) && a.first == b.first && a.last == b.last && a.empty == b.empty &&
           same(a.prefix, b.prefix) && same(a.suffix, b.suffix) && same(a.best, b.best);
}

float value(std::mt19937_64& rng, int kind) {
    constexpr float kInf = std::numeric_limits<float>::infinity(), kNan = std::numeric_limits<float>::quiet_NaN();
    constexpr float kTiny = std::numeric_limits<float>::denorm_min();
    const float sign = rng() % 2 == 0 ? 1.0F : -1.0F;
    switch (kind) {
    case 0: return sign * static_cast<float>(rng() % 3);         // +-0, ties, exact cancellation
    case 1: return sign * kTiny * static_cast<float>(rng() % 4); // multiples of 2^-149
    case 2: return std::normal_distribution<float>(0.0F, 1.0F)(rng);
    case 3: return rng() % 6 == 0 ? std::copysign(kNan, sign) : sign * static_cast<float>(rng() % 4);
    case 4: return rng() % 8 == 0 ? sign * kInf : sign * static_cast<float>(rng() % 4);
    default: return rng() % 3 == 0 ? sign * kTiny : sign * std::ldexp(1.0F, static_cast<int>(rng() % 250) - 125);
    }
}

} // namespace

int main() {
    std::mt19937_64 rng(512);
    long bad = 0, cases = 0;
    for (int trial = 0; trial < 200000; ++trial, ++cases) {
        const int n     = static_cast<int>(rng() % 40), kind = static_cast<int>(rng() % 6);
        const int first = static_cast<int>(rng() % 5);
        KadaneState time_pos = KadaneState::make(), time_neg = KadaneState::make();
        KadaneState row_pos = KadaneState::make(), row_neg = KadaneState::make();
        KadanePair32 pair;
        KadaneBest pos, neg;
        if (n > 0)
            pair.begin(first);
        for (int i = first; i < first + n; ++i) {
            const double u  = value(rng, kind);
            const bool used = rng() % 4 != 0;
            time_pos.append(i, u);
            time_neg.append(i, -u);
            pair.append(i, u);
            if (used) {
                row_pos.append(i, u);
                row_neg.append(i, -u);
            }
            pos.append(i, used ? u : 0.0);
            neg.append(i, used ? -u : -0.0);
        }
        auto best = [](const KadaneBest& b, const KadaneState& full) {
            return full.best.length() > 0 ? same(b.best(), full.best) : b.best().length() <= 0;
        };
        if (!same(pair.widen_pos(first + n - 1), time_pos) || !same(pair.widen_neg(first + n - 1), time_neg) ||
            !best(pos, row_pos) || !best(neg, row_neg))
            ++bad;
    }
    std::printf("cases %ld bad %ld\n", cases, bad);
    return bad == 0 ? 0 : 1;
}
