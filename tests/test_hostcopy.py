"""Copies of pageable arrays through page-locked slots (csrc/hostcopy.h) on the
CPU: a small harness is compiled against it with host memory for the device's
and the CUDA runtime's few calls answered at once."""
import os
import subprocess

import pytest

from conftest import PKG

HARNESS = r"""
#include <dirent.h>
#include <signal.h>
#include <stdlib.h>
#include <string.h>
#include <sys/resource.h>
#include <sys/wait.h>
#include <unistd.h>
#include <cstdio>
#include <vector>
#include "hostcopy.h"

static bool g_no_pin = false;
extern "C" {
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
    memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = reinterpret_cast<cudaEvent_t>(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) {
    if (g_no_pin) return cudaErrorMemoryAllocation;
    return (*p = malloc(n)) ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaHostRegister(void *, size_t, unsigned) { return g_no_pin ? cudaErrorMemoryAllocation : cudaSuccess; }
cudaError_t cudaHostUnregister(void *) { return cudaSuccess; }
}

using sarbp::HostStager;

static int threads() {
    int n = 0;
    DIR *d = opendir("/proc/self/task");
    while (dirent *e = readdir(d)) n += e->d_name[0] != '.';
    closedir(d);
    return n;
}
static double cpu_seconds() {
    rusage r;
    getrusage(RUSAGE_SELF, &r);
    return r.ru_utime.tv_sec + r.ru_stime.tv_sec + 1e-6 * (r.ru_utime.tv_usec + r.ru_stime.tv_usec);
}
// kB of mappings that a forked child does not get
static long kept_from_children() {
    FILE *f = fopen("/proc/self/smaps", "r");
    char line[4096];
    long size = 0, total = 0;
    while (fgets(line, sizeof(line), f)) {
        sscanf(line, "Size: %ld kB", &size);
        if (!strncmp(line, "VmFlags:", 8) && strstr(line, " dc")) total += size;
    }
    fclose(f);
    return total;
}
// n bytes up and down again; whether they arrived
static bool round_trip(HostStager &s, size_t n, unsigned seed) {
    std::vector<char> a(n), dev(n), b(n);
    for (size_t i = 0; i < n; ++i) a[i] = (char)((i * 2654435761u + seed) >> 13);
    HostStager::Session session(&s);
    if (s.upload(dev.data(), a.data(), n, nullptr) != cudaSuccess) return false;
    if (dev != a) return false;
    return s.download(b.data(), dev.data(), n, nullptr) == cudaSuccess && s.drain() == cudaSuccess && b == a;
}

int main(int, char **argv) {
    alarm(60);
    HostStager *s = new HostStager;
    bool ok = true;
    if (!strcmp(argv[1], "data")) {
        const size_t sizes[] = {1, 128 << 10, (128 << 10) + 1, (2 << 20) - 1, 2 << 20, (2 << 20) + 4097, 40000003};
        for (int rep = 0; rep < 20; ++rep)
            for (size_t n : sizes) ok = ok && round_trip(*s, rep < 10 || n < (3 << 20) ? n : 1000, rep);
    } else if (!strcmp(argv[1], "nothing_staged")) {
        HostStager::Session session(s);
        ok = threads() == 1;
    } else if (!strcmp(argv[1], "idle")) {
        std::vector<char> a(8 << 20, 1), dev(8 << 20);
        HostStager::Session session(s);
        ok = s->upload(dev.data(), a.data(), a.size(), nullptr) == cudaSuccess;
        const double t = cpu_seconds();
        usleep(500000);  // a kernel runs
        ok = ok && cpu_seconds() - t < 0.1;
        ok = ok && round_trip(*s, 9000001, 5);
    } else if (!strcmp(argv[1], "fork")) {
        ok = round_trip(*s, 9000001, 1);
        usleep(100000);  // the threads sleep
        const pid_t c = fork();
        if (c == 0) {
            const bool good = round_trip(*s, 9000001, 2);
            delete s;
            _exit(good ? 0 : 1);
        }
        int st = 0, k = 0;
        while (waitpid(c, &st, WNOHANG) == 0 && k++ < 100) usleep(100000);
        if (k > 100) {
            kill(c, SIGKILL);
            waitpid(c, &st, 0);
            std::printf("the child hangs\n");
            return 1;
        }
        ok = ok && WIFEXITED(st) && WEXITSTATUS(st) == 0 && round_trip(*s, 9000001, 3);
    } else if (!strcmp(argv[1], "slots_stay_out_of_a_child")) {
        ok = round_trip(*s, 9000001, 6);
        ok = ok && kept_from_children() >= (16 << 10);
    } else if (!strcmp(argv[1], "no_page_locked_memory")) {
        g_no_pin = true;
        ok = round_trip(*s, 9000001, 4);
        g_no_pin = false;
        ok = ok && round_trip(*s, 9000001, 5);
    }
    s->release();
    delete s;
    std::printf("%s\n", ok ? "ok" : "wrong");
    return ok ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    cuda_inc = "/usr/local/cuda/include"
    if not os.path.isdir(cuda_inc):
        pytest.skip("CUDA headers not found")
    d = tmp_path_factory.mktemp("hostcopy")
    src, out = d / "harness.cpp", str(d / "harness")
    src.write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", os.path.join(PKG, "csrc"), "-I", cuda_inc, str(src),
                    os.path.join(PKG, "csrc", "hostcopy.cpp"), "-o", out], check=True)
    return out


@pytest.mark.parametrize("what", ["data", "fork", "nothing_staged", "idle", "no_page_locked_memory",
                                  "slots_stay_out_of_a_child"])
def test_staged_copies(exe, what):
    """The bytes arrive; a forked child copies by itself and may drop the
    object; threads start with the first staged copy and sleep while nothing is
    copied; without page-locked memory the copies are the driver's; a fork does
    not make the slots' pages copies-on-write, under which the device would
    go on with the old pages."""
    p = subprocess.run([exe, what], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0 and p.stdout.strip() == "ok", p.stdout
