// Values per device (nricp_b200/csrc/per_device.hpp): see tests/test_per_device.py.
#include <cstdio>
#include <stdexcept>
#include <thread>
#include <vector>

#include "../nricp_b200/csrc/per_device.hpp"

int main() {
    int failures = 0;
    auto expect = [&](bool ok, const char* what) {
        if (ok) return;
        ++failures;
        std::printf("%s\n", what);
    };
    nricp_b200::PerDevice<int> values;
    int made[2] = {0, 0};
    auto value = [&](int device) -> const int& {
        return values.of(device, [&] { return 10 * device + ++made[device]; });
    };
    const int& first = value(0);
    expect(first == 1 && value(0) == 1 && made[0] == 1, "made once on the first device");
    expect(value(1) == 11 && made[1] == 1, "made again on the second device");
    expect(&value(0) == &first, "references stay valid");
    nricp_b200::PerDevice<int> refused;
    bool thrown = false;
    try {
        refused.of(0, []() -> int { throw std::runtime_error("refused"); });
    } catch (const std::runtime_error&) {
        thrown = true;
    }
    expect(thrown && refused.of(0, [] { return 7; }) == 7, "a failure is not kept");
    nricp_b200::PerDevice<int> shared;
    int runs = 0;  // under the value's own lock
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&] {
            for (int i = 0; i < 1000; ++i) shared.of(i % 4, [&] { return ++runs; });
        });
    for (std::thread& t : threads) t.join();
    expect(runs == 4, "made once per device by several threads");
    std::printf(failures ? "FAILED\n" : "ok\n");
    return failures ? 1 : 0;
}
