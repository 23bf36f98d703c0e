// csrc/once.h on host threads: nobody goes on before the preparation is done, it is done once per device, and a failed one is
// tried again.  Exit code 0 if all of that holds.
#include <chrono>
#include <thread>
#include <vector>

#include "once.h"

int main() {
    static vdnn::OncePerDevice once;
    std::atomic<int> runs[3], ready[3], early(0), failures(0);
    for (int d = 0; d < 3; ++d) runs[d] = ready[d] = 0;
    std::vector<std::thread> threads;
    for (int t = 0; t < 12; ++t)
        threads.emplace_back([&, t] {
            const int d = t % 3;
            auto prepare = [&] {
                std::this_thread::sleep_for(std::chrono::milliseconds(20));
                if (++runs[d] == 1 && d == 2) return 7;             // the first attempt on device 2 fails
                ready[d] = 1;
                return 0;
            };
            const int status = once.run(d, prepare);
            if (status == 7) ++failures;
            else if (status != 0 || !ready[d]) ++early;
        });
    for (auto& t : threads) t.join();
    if (early != 0) return 1;
    if (runs[0] != 1 || runs[1] != 1) return 2;
    if (failures != 1 || runs[2] != 2) return 3;
    int beyond = 0;
    for (int i = 0; i < 2; ++i)
        if (once.run(100, [&] { ++beyond; return 0; }) != 0) return 4;
    return beyond == 2 ? 0 : 5;
}
