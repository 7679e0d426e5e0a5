// Prints what the host-side dispatch of sf_api.cu decides, one line per line of
// standard input, for the tests that need no GPU.  Plans are made here, for a
// device of 152 SMs, with field pointers that nothing dereferences.
//
// The state-on-chip launches run here too, against calls that are only listed.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <iostream>
#include <sstream>
#include <string>

namespace probe {

std::string calls;        // what was called, in order
int launches_left = 1000;  // launches that succeed
size_t room = size_t(1) << 30;  // largest allocation that succeeds

cudaError_t note(const char* what) {
    calls += what;
    calls += ' ';
    return cudaSuccess;
}
template <class T>
cudaError_t malloc(T** p, size_t bytes) {
    if (bytes > room) return cudaErrorMemoryAllocation;
    *p = reinterpret_cast<T*>(uintptr_t(1) << 20);
    return note("malloc");
}

template <class... A>
cudaError_t launch(const cudaLaunchConfig_t* cfg, A...) {
    return note(cfg->numAttrs > 0 ? "dependent" : "plain");
}

}  // namespace probe

#define cudaStreamWaitEvent(...) probe::note("wait")
#define cudaEventRecord(...) probe::note("record")
#define cudaMalloc(...) probe::malloc(__VA_ARGS__)
#define cudaFree(...) probe::note("free")
#define cudaMemsetAsync(...) probe::note("clear")
#define cudaThreadExchangeStreamCaptureMode(...) probe::note("mode")
#define cudaLaunchKernelEx(...) probe::launch(__VA_ARGS__)
#define cudaHostAlloc(p, n, ...) (*(p) = ::calloc(1, n), cudaSuccess)
#define cudaHostGetDevicePointer(d, h, ...) (*(d) = (h), cudaSuccess)
#define cudaEventCreateWithFlags(e, ...) (*(e) = reinterpret_cast<cudaEvent_t>(uintptr_t(4096)), cudaSuccess)
#define cudaGetDevice(d) (*(d) = 0, cudaSuccess)
#define cudaMallocAsync(p, n, ...) probe::malloc(p, n)
#define cudaFreeAsync(...) probe::note("free-behind")
#define cudaMemcpyAsync(...) probe::note("copy")
#define cudaStreamSynchronize(...) probe::note("sync")
#include "sf_api.cu"
#include "sf_step.cu"
#include "sf_voxel.cu"

int sf_launch_step_tile_cfg(const SfStepArgs&, const SfSources&, bool, int cfg, int, cudaStream_t) {
    probe::note(kSfTileConfigs[cfg].name);
    return 0;
}
int sf_launch_step_tb(const SfStepArgs&, const SfSources&, bool, int cfg, int, float*, cudaStream_t) {
    probe::note(kSfTbConfigs[cfg].name);
    return 0;
}
int sf_launch_resident(SfResArgs&, const SfSources&, const SfResCut&, cudaStream_t) {
    probe::note("launch");
    return --probe::launches_left >= 0 ? 0 : sf_fail("launch failed");
}

namespace {

constexpr int kSms = 152;

sf_plan plan_of(int nx, int ny, int nz, bool walls) {
    sf_plan P;
    P.d.nx = nx;
    P.d.ny = ny;
    P.d.nz = nz;
    P.n = (long long)nx * ny * nz;
    P.sms = kSms;
    for (auto& set : P.f)
        for (auto& f : set) f = reinterpret_cast<float*>(uintptr_t(4096));
    if (walls) P.flags = reinterpret_cast<uint8_t*>(uintptr_t(4096));
    return P;
}

void cut(std::istringstream& in) {  // nx ny nz probes nu planes: the state-on-chip cut
    int nx, ny, nz, probes, nu, planes;
    in >> nx >> ny >> nz >> probes >> nu >> planes;
    SfResExtra x{};
    x.n_plane = planes;
    for (int q = 0; q < planes; ++q) x.ops[q].axis = q % 3;
    const SfResCut c = sf_resident_cut(nx, ny, nz, probes, nu != 0, kSms, planes ? &x : nullptr);
    std::printf("%d %d %d %d %d %d\n", c.kind, c.bi, c.bj, c.bk, c.side_max, c.threads);
}

void pair(std::istringstream& in) {  // nx ny nz walls plane_axis: the two-step choice
    int nx, ny, nz, walls, axis;
    in >> nx >> ny >> nz >> walls >> axis;
    sf_plan P = plan_of(nx, ny, nz, walls != 0);
    P.src.n = 1;
    P.src.s[0].kind = axis >= 0;
    P.src.s[0].a = axis >= 0 ? axis : 1;
    SfStepArgs a;
    fill_args(&P, a, false);
    set_io(&P, a, 0);
    const int c = default_pair(&P, a);
    std::printf("%s\n", c < 0 ? "-" : sf_kernel_config_name(c));
}

void weighted(std::istringstream& in) {  // nx ny nz, cells: whether the plan may stay on the chip
    int nx, ny, nz;
    in >> nx >> ny >> nz;
    sf_plan P = plan_of(nx, ny, nz, false);
    std::vector<int64_t> cells;
    for (int64_t c; in >> c;) cells.push_back(c);
    const std::vector<double> w(cells.size(), 1.0);
    sf_plan_set_weighted_source(&P, 0, (int64_t)cells.size(), cells.data(), w.data());
    P.wsrc_n[0] = (long long)cells.size();  // (without a device the tables' copies fail)
    P.src.n = 1;
    P.src.s[0].kind = 2;
    SfResExtra x;
    std::printf("%d\n", resident_extra(&P, false, x) ? 1 : 0);
}

void steps(std::istringstream& in) {  // nx ny nz, steps, launches that succeed: the calls made
    int nx, ny, nz, n;
    in >> nx >> ny >> nz >> n >> probe::launches_left;
    sf_plan P = plan_of(nx, ny, nz, false);
    SfStepArgs a;
    fill_args(&P, a, false);
    P.res_cut = sf_resident_cut(nx, ny, nz, 0, false, kSms, nullptr);
    g_res[0].done = reinterpret_cast<cudaEvent_t>(uintptr_t(4096));
    probe::calls.clear();
    const int rc = step_resident(&P, a, n, nullptr, nullptr, nullptr, nullptr);
    std::printf("%s%d\n", probe::calls.c_str(), rc);
}

int config_named(const std::string& name) {
    for (int q = 0; q < sf_kernel_config_count(); ++q)
        if (name == sf_kernel_config_name(q)) return q;
    return -1;
}

// nx ny nz walls plane_axis, the tuned configuration ("-": none), steps: their kernels
void tuned(std::istringstream& in) {
    int nx, ny, nz, walls, axis, n;
    std::string name;
    in >> nx >> ny >> nz >> walls >> axis >> name >> n;
    sf_plan P = plan_of(nx, ny, nz, walls != 0);
    P.bound = true;
    P.tuned = name == "-" ? 0 : config_named(name);
    P.src.n = 1;
    P.src.s[0].kind = axis >= 0;
    P.src.s[0].a = axis >= 0 ? axis : 1;
    const double value = 0.0;
    probe::calls.clear();
    const int rc = sf_plan_step(&P, n, &value, nullptr, nullptr);
    std::printf("%s%d\n", probe::calls.c_str(), rc);
}

// nx ny nz: the calls of a mask (without a device its kernels fail to launch) and
// whether its scratch memory may be lent again
void mask(std::istringstream& in) {
    int nx, ny, nz;
    in >> nx >> ny >> nz;
    sf_sdf_node ball{};
    ball.op = 2;
    ball.s0 = 1.0;
    probe::calls.clear();
    const int rc = sf_voxelize(&ball, 1, nx, ny, nz, 0.1, 0, reinterpret_cast<uint8_t*>(uintptr_t(4096)),
                               nullptr);
    std::printf("%s%s%d\n", probe::calls.c_str(), g_keep[0].lent ? "lent " : "", rc);
}

void ade(std::istringstream& in) {  // density poles, modulus poles, serial: the launches of a step
    SfPoles poles{};
    int serial;
    in >> poles.n_density >> poles.n_modulus >> serial;
    poles.n = poles.n_density + poles.n_modulus;
    sf_plan P = plan_of(20, 20, 80, false);
    for (int q = 0; q < 3; ++q) P.ade_hi[q] = 10;
    SfStepArgs a;
    fill_args(&P, a, false);
    a.serial = serial;
    probe::calls.clear();
    const int rc = sf_launch_step(a, SfSources{}, poles, false, nullptr);
    std::printf("%s%d\n", probe::calls.c_str(), rc);
}

}  // namespace

int main() {
    std::string line, what;
    while (std::getline(std::cin, line)) {
        std::istringstream in(line);
        in >> what;
        if (what == "cut") cut(in);
        else if (what == "pair") pair(in);
        else if (what == "weighted") weighted(in);
        else if (what == "steps") steps(in);
        else if (what == "tuned") tuned(in);
        else if (what == "mask") mask(in);
        else if (what == "room") in >> probe::room;
        else if (what == "ade") ade(in);
        else return 2;
    }
    return 0;
}
