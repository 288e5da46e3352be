// CPU check of WaitOnThrow (faz_gb300/csrc/host.h) against a counting stand-in for
// cudaStreamSynchronize: a scope left by an exception waits for its stream before the
// exception goes on, inner scopes before outer ones, also inside a handler; a scope
// left otherwise does not wait.
#include <cstdio>
#include <stdexcept>

#include "../faz_gb300/csrc/host.h"

static std::vector<cudaStream_t> waited;
extern "C" cudaError_t CUDARTAPI cudaStreamSynchronize(cudaStream_t st) {
    waited.push_back(st);
    return cudaSuccess;
}
extern "C" cudaError_t CUDARTAPI cudaFreeHost(void *) { return cudaSuccess; }
extern "C" cudaError_t CUDARTAPI cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }

static int failures = 0;
static void expect(const char *what, std::vector<cudaStream_t> want) {
    if (waited != want) {
        std::printf("%s: %zu waits, %zu expected\n", what, waited.size(), want.size());
        failures++;
    }
    waited.clear();
}

int main() {
    int a, b;
    const cudaStream_t A = reinterpret_cast<cudaStream_t>(&a), B = reinterpret_cast<cudaStream_t>(&b);
    {
        faz::WaitOnThrow w(A);
    }
    expect("left at its end", {});
    auto f = [&](bool fail) {
        faz::WaitOnThrow w(A);
        if (!fail) return;
        faz::WaitOnThrow v(B);
        throw faz::Fail{-4, "damaged"};
    };
    f(false);
    expect("left by return", {});
    try {
        f(true);
    } catch (const faz::Fail &) {
        expect("left by an exception", {B, A});
        // a handler's own scopes: the exception behind it does not count
        f(false);
        expect("a handler, left by return", {});
        try {
            f(true);
        } catch (...) {
            expect("a handler, left by an exception", {B, A});
        }
    }
    try {
        faz::WaitOnThrow w(A);
        try {
            throw std::runtime_error("handled");
        } catch (const std::exception &) {
        }
        expect("handled inside", {});
    } catch (...) {
        failures++;
    }
    expect("left at its end after a handled one", {});
    return failures != 0;
}
