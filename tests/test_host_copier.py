"""The host copier (csrc/host_copy.cuh) against a stand-in for the CUDA
runtime, on the CPU: what its copies do around its piece size, after a set-up
that the runtime refused, and in which capture mode its threads wait.  In the
stand-in a transfer runs only when an event recorded behind it is waited for,
or at the end, so a buffer that is written too early shows in the data."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "nimbus_b200" / "csrc"
CUDA_INCLUDE = next((p for p in ("/usr/local/cuda/include",) if Path(p, "cuda_runtime.h").exists()), None)

PROGRAM = r"""
#include "host_copy.cuh"
#include <cstdio>
#include <cstdlib>
#include <deque>
#include <functional>
#include <map>
#include <string>

static std::mutex lock;
static std::deque<std::pair<int, std::function<void()>>> queue;  // transfers, by their number
static std::map<cudaEvent_t, int> recorded;
static int enqueued = 0, refuse_pinned = 0;
static thread_local cudaStreamCaptureMode mode = cudaStreamCaptureModeGlobal;
static std::atomic<int> strict_waits{0};

static void run_to(int number)
{
    while (!queue.empty() && queue.front().first <= number)
    {
        queue.front().second();
        queue.pop_front();
    }
}

extern "C" {
cudaError_t cudaMallocHost(void** p, size_t n)
{
    if (refuse_pinned > 0 && refuse_pinned--) return cudaErrorMemoryAllocation;
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned)
{
    *e = reinterpret_cast<cudaEvent_t>(std::malloc(1));
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t)
{
    std::lock_guard<std::mutex> g(lock);
    recorded[e] = enqueued;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
    std::lock_guard<std::mutex> g(lock);
    if (mode != cudaStreamCaptureModeRelaxed) ++strict_waits;
    run_to(recorded[e]);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    std::lock_guard<std::mutex> g(lock);
    queue.emplace_back(++enqueued, [=] { std::memcpy(d, s, n); });
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m) { std::swap(*m, mode); return cudaSuccess; }
}

using nimbus_host::HostCopier;
static void flush() { std::lock_guard<std::mutex> g(lock); run_to(enqueued); }
static int failures = 0;
#define EXPECT(x) do { if (!(x)) { std::printf("failed: %s (line %d)\n", #x, __LINE__); ++failures; } } while (0)

static void sizes(HostCopier& c)
{
    const size_t piece = HostCopier::kPiece;
    for (size_t n : {piece, 4 * piece, 4 * piece + 1, 9 * piece - 3, 40 * piece + 17})
    {
        std::vector<char> host(n), device(n), back(n);
        for (size_t i = 0; i < n; ++i) host[i] = (char)(i * 31 + i / piece);
        cudaError_t result = cudaErrorUnknown;
        EXPECT(c.copy(true, device.data(), host.data(), n, nullptr, &result) && result == cudaSuccess);
        std::vector<char> sent = host;
        std::fill(host.begin(), host.end(), 0);  // the caller may reuse its array
        flush();
        EXPECT(device == sent);
        EXPECT(c.copy(false, device.data(), back.data(), n, nullptr, &result) && result == cudaSuccess);
        EXPECT(back == sent);
    }
}

int main(int, char** argv)
{
    const std::string what = argv[1];
    if (what == "setup")
    {
        refuse_pinned = 1;
        EXPECT(!HostCopier::of_device(0, false));
        EXPECT(!HostCopier::of_device(0, true));  // refused: the caller copies the ordinary way
        std::shared_ptr<HostCopier> c = HostCopier::of_device(0, true);
        EXPECT(c && c->ready());
        EXPECT(HostCopier::of_device(0, false) == c);
        return failures;
    }
    HostCopier c(0);
    EXPECT(c.ready());
    if (what == "sizes") sizes(c);
    if (what == "mode")
    {
        cudaStreamCaptureMode relaxed = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&relaxed);  // as the caller chose for its own thread
        sizes(c);
        EXPECT(strict_waits == 0);
    }
    return failures;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if CUDA_INCLUDE is None or shutil.which("g++") is None:
        pytest.skip("needs g++ and the CUDA headers")
    folder = tmp_path_factory.mktemp("copier")
    (folder / "copier.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-x", "c++", "copier.cpp", "-I", str(CSRC), "-I", CUDA_INCLUDE, "-o",
                    "copier", "-pthread"], cwd=folder, check=True)
    return folder / "copier"


@pytest.mark.parametrize("what", ["sizes", "setup", "mode"])
def test_copier(program, what):
    done = subprocess.run([program, what], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, done.stdout
