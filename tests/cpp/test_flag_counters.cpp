// The number that counts a launch's finished CTAs (flag_counters.h), through
// every order in which the CTAs of one launch, and of two or three that overlap,
// can add to it and take a launch's CTAs out again: the count ends at zero, each
// launch has one last CTA, and the settled windows are those of all CTAs.
#include <cstdio>

#include "flag_counters.h"

namespace {

constexpr uint32_t kCtas = 3;
long orders = 0;
bool ok = true;

// left: CTAs that have not added yet; due: launches to be taken out
void step(uint64_t number, uint32_t left, uint32_t launches, int due, uint32_t lasts)
{
    if (left == 0 && due == 0) {
        ++orders;
        uint64_t settled = 0;
        for (uint32_t k = 1; k <= launches * kCtas; ++k) settled += k;
        ok = ok && number == settled << opiv::kDoneBits && lasts == launches;
        return;
    }
    if (left > 0) {
        const bool last = opiv::last_done(number, kCtas);
        ok = ok && opiv::all_settled(number, left) == (number + opiv::done_add(left)) >> opiv::kDoneBits;
        step(number + opiv::done_add(left), left - 1, launches, due + last, lasts + last);   // `left` settled windows
    }
    if (due > 0) step(number - kCtas, left, launches, due - 1, lasts);
}

}  // namespace

int main()
{
    for (uint32_t launches = 1; launches <= 3; ++launches) step(0, launches * kCtas, launches, 0, 0);
    if (!ok) return 1;
    std::printf("ok %ld orders\n", orders);
    return 0;
}
