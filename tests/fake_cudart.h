// Controls and counters of the fake CUDA runtime.
#pragma once
#include <atomic>
namespace fake {
extern std::atomic<long long> device_bytes;    // allocated now
extern std::atomic<long long> device_limit;    // most that may be allocated (-1: no limit)
extern std::atomic<long long> host_limit;      // largest pinned buffer (-1: no limit)
extern std::atomic<int> copies;                // copies enqueued so far
extern std::atomic<int> fail_copy;             // number of the copy that fails (-1: none)
extern std::atomic<int> stream_syncs;
extern std::atomic<int> open_copies;           // enqueued since the last stream synchronisation
}
