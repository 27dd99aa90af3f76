// The wait of report_wait.cuh against a stream that is played by a function.
#include <cstdio>

#include "../../dmtz_gb300/csrc/report_wait.cuh"

int main() {
    int bad = 0;
    auto check = [&](const char *what, cudaError_t got, cudaError_t want) {
        if (got == want) return;
        printf("%s: %d, want %d\n", what, (int)got, (int)want);
        bad++;
    };
    unsigned long long at = 5;
    int calls = 0;
    auto never = [&]() { calls++; return cudaErrorNotReady; };
    check("written before", dmtz::wait_report(&at, 5, never), cudaSuccess);
    bad += calls != 0;
    auto later = [&]() {
        if (++calls == 3) at = 6;
        return cudaErrorNotReady;
    };
    check("written while the stream runs", dmtz::wait_report(&at, 6, later), cudaSuccess);
    auto last = [&]() {
        at = 7;
        return cudaSuccess;
    };
    check("written just before the stream is idle", dmtz::wait_report(&at, 7, last), cudaSuccess);
    check("idle, not written", dmtz::wait_report(&at, 8, []() { return cudaSuccess; }), cudaErrorUnknown);
    check("failed", dmtz::wait_report(&at, 8, []() { return cudaErrorLaunchFailure; }), cudaErrorLaunchFailure);
    printf("%d wrong\n", bad);
    return bad != 0;
}
