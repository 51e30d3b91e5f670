// Host-side checks of the plan's numbers that place an access (rsbd8g::plan_in_range, prefix_in_range): what
// plan_chain writes for every set of digits passes them and stays within the plan, and what names no digit or
// look-back array of the key, or no pass slot, does not.  Built with nvcc, run on the host (no GPU needed).
#include <cstdio>

#include "rsbd8g_prefix.cuh"

using namespace rsbd8g;

static int failures = 0;
static void check(bool ok, const char *what) {
    if (!ok) {
        std::printf("FAIL: %s\n", what);
        ++failures;
    }
}

template <int DIGITS>
static void key_of() {
    uint32_t hot[kMaxPasses];
    for (uint32_t &h : hot) h = kNoHotPair;
    PlanArgs a{};
    a.passes = DIGITS;
    for (uint32_t survive = 1; survive < (1u << DIGITS); survive += DIGITS > 10 ? 37u : 1u) {
        for (int failed = 0; failed < 2; ++failed) {       // the passes of the plan, and those after a failed settle step
            Control c{};
            uint32_t curk = kArrKeysA;
            plan_chain(&c, a, hot, survive, failed != 0, failed ? kPrefixSlots : 0, kArrIn, curk, false, false);
            uint32_t seen = 0;
            for (int s = 0; s < kMaxSlots; ++s) {
                if (!c.plan[s].active) continue;
                check(plan_in_range<DIGITS>(c.plan[s]), "a planned pass is in range");
                check(s < DIGITS + (failed ? kPrefixSlots : 0), "a planned pass has a launch");
                seen |= 1u << c.plan[s].digit;
            }
            check(seen == survive, "every surviving digit is planned");
        }
    }
    PassPlan p{};
    for (uint32_t v : {uint32_t(DIGITS), uint32_t(DIGITS) + 1u, 0x100u, 0xFFFFu}) {
        p.digit = uint16_t(v), p.status = 0;
        check(!plan_in_range<DIGITS>(p), "a digit the key does not have");
        p.digit = 0, p.status = uint16_t(v);
        check(!plan_in_range<DIGITS>(p), "a look-back array the sort does not have");
    }
    const uint32_t all = (1u << DIGITS) - 1u;
    check(prefix_in_range<DIGITS>(0, 0, 0) && prefix_in_range<DIGITS>(kPrefixSlots, DIGITS - 1, all), "prefixes in range");
    check(!prefix_in_range<DIGITS>(kPrefixSlots + 1, 0, all) && !prefix_in_range<DIGITS>(0xFFFFFFFFu, 0, all), "too many passes");
    check(!prefix_in_range<DIGITS>(1, DIGITS, all), "a lowest digit the key does not have");
    check(!prefix_in_range<DIGITS>(1, 0, all + 1u) && !prefix_in_range<DIGITS>(1, 0, 0x80000001u), "digits the key does not have");
}

int main() {
    key_of<8>();
    key_of<10>();
    key_of<16>();
    if (failures == 0) std::printf("ok\n");
    return failures == 0 ? 0 : 1;
}
