// tune_pin.cpp -- host check of the tuning table's versions (runtime.cu): a
// pinned thread keeps reading the table its pin was made with while another
// thread sets, loads and clears knobs.  Prints "ok", or the first failure
// (exit code 1).
#include <cstdio>
#include <thread>

#include "runtime.cuh"

using namespace zk;

#define CHECK(x)                                       \
    do {                                               \
        if (!(x)) {                                    \
            printf("line %d: %s\n", __LINE__, #x);     \
            return 1;                                  \
        }                                              \
    } while (0)

int main(int, char **argv)
{
    tune_clear();
    tune_set("ntt_split_logr", TUNE_ANY, 9);
    const uint64_t gen = tune_generation();
    TuneVersion queued;
    {
        TunePin pin;
        queued = tune_version();
        std::thread([&] {
            tune_set("ntt_split_logr", TUNE_ANY, 7);
            tune_load_file(argv[1]);  // "ntt_split_logr 12 10"
        }).join();
        CHECK(tune_get("ntt_split_logr", 12, 0) == 9 && tune_generation() == gen);
        {
            TunePin inner;  // keeps the enclosing pin's version
            CHECK(tune_get("ntt_split_logr", 12, 0) == 9);
        }
        CHECK(tune_get("ntt_split_logr", 12, 0) == 9);
        tune_set("ntt_split_logr", TUNE_ANY, 8);  // this thread's own change too
        CHECK(tune_get("ntt_split_logr", 13, 0) == 9 && tune_generation() == gen);
    }
    CHECK(tune_get("ntt_split_logr", 13, 0) == 8 && tune_get("ntt_split_logr", 12, 0) == 10);
    CHECK(tune_generation() == gen + 3);
    tune_clear();
    {
        TunePin pin(queued);  // a queued request's version outlives the changes
        CHECK(tune_get("ntt_split_logr", 12, 0) == 9 && tune_generation() == gen);
    }
    CHECK(tune_get("ntt_split_logr", 12, 0) == 0);
    {
        TunePin outer;  // reads nothing before the inner pin does
        {
            TunePin inner;
            CHECK(tune_get("ntt_split_logr", 12, 0) == 0);
            {
                TunePin request(queued);
                CHECK(tune_get("ntt_split_logr", 12, 0) == 9);
            }
        }
        tune_set("ntt_split_logr", 12, 5);
        CHECK(tune_get("ntt_split_logr", 12, 0) == 0);
    }
    CHECK(tune_get("ntt_split_logr", 12, 0) == 5);
    // readers of one version see one value however often it changes
    bool same = true, stop = false;
    std::thread writer([&] {
        for (uint64_t v = 1; v < 20000; v++) tune_set("ntt_split_logr", 12, v);
        __atomic_store_n(&stop, true, __ATOMIC_RELEASE);
    });
    while (!__atomic_load_n(&stop, __ATOMIC_ACQUIRE)) {
        TunePin pin;
        const uint64_t a = tune_get("ntt_split_logr", 12, 0);
        std::this_thread::yield();
        same = same && tune_get("ntt_split_logr", 12, 0) == a;
    }
    writer.join();
    CHECK(same);
    printf("ok\n");
    return 0;
}
