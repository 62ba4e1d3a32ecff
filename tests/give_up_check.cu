// Test harness (GPU): a resident run or search whose barrier gives up must end
// with a status and leave a context that a new state makes usable. Linked with
// the library's own objects, so that it can write the barrier's words. Built
// and run by tests/test_gpu_give_up.py; returns 0, or the number of the check
// that failed.
#include <cstring>
#include <vector>

#include "../cubble_gb300/csrc/context.cuh"

using namespace cbg;

namespace {

struct Pairs {
    std::vector<int> i, j;
    bool get(cb_context *c) {
        int n = 0;
        i.assign(c->hk.pcap, 0);
        j.assign(c->hk.pcap, 0);
        if (cb_get_pairs(c, i.data(), j.data(), c->hk.pcap, &n)) return false;
        i.resize(n);
        j.resize(n);
        return n > 0;
    }
};

bool set_arrivals(cb_context *c, unsigned v) {
    return cudaMemcpy(&c->bufs.run->arrive, &v, sizeof v, cudaMemcpyHostToDevice) == cudaSuccess;
}

bool sync_is_clear(cb_context *c) {
    RunSync s, zero;
    std::memset(&zero, 0, sizeof zero);
    return cudaMemcpy(&s, c->bufs.run, sizeof s, cudaMemcpyDeviceToHost) == cudaSuccess &&
           std::memcmp(&s, &zero, sizeof s) == 0;
}

int usable_again(cb_context *c, const cb_state_view *st, const Pairs &want) {
    Pairs p;
    cb_report r;
    if (cb_load_state(c, st)) return 1;
    if (cb_search_neighbors(c)) return 2;
    if (!p.get(c) || p.i != want.i || p.j != want.j) return 3;
    if (cb_bootstrap(c) || cb_integrate(c, 3, &r) || r.status != CB_OK) return 4;
    return 0;
}

}  // namespace

extern "C" __attribute__((visibility("default"))) int give_up(const cb_config *cfg,
                                                              const cb_state_view *st) {
    cb_context *c = nullptr;
    Pairs want;
    if (cb_create(cfg, &c) || cb_load_state(c, st) || cb_search_neighbors(c) || !want.get(c))
        return 1;

    // A grid that lacks one of its blocks: with one arrival in advance the
    // search passes its first barrier and waits at the second until its limit
    // (seconds); the cells are counted by then, so the counts are left behind.
    const int blocks = 12;
    std::vector<RunBlock> map;
    for (int v = 0; v < blocks; v++) map.push_back({0, v, blocks + 1});
    RunBlock *dmap = nullptr;
    Bufs *dbufs = nullptr;
    if (cb_load_state(c, st) || cudaMalloc(&dmap, sizeof(RunBlock) * blocks) ||
        cudaMalloc(&dbufs, sizeof(Bufs)) ||
        cudaMemcpy(dmap, map.data(), sizeof(RunBlock) * blocks, cudaMemcpyHostToDevice) ||
        cudaMemcpy(dbufs, &c->bufs, sizeof(Bufs), cudaMemcpyHostToDevice))
        return 2;
    if (c->pull()) return 3;
    c->hctrl->bsel = SEL_SEARCH;
    if (c->push() || !set_arrivals(c, 1)) return 3;
    RunLaunch r;
    r.grid = blocks;
    r.block = kBlock;
    r.stream = c->stream;
    r.steps = 1;
    r.mirror = nullptr;
    r.launches = &c->launches;
    r.foams = dbufs;
    r.map = dmap;
    launch_search_run(r, c->bufs, c->hk.dim);
    if (cudaStreamSynchronize(c->stream) != cudaSuccess || c->pull()) return 4;
    if (c->hctrl->status != CB_ERR_CUDA) return 5;
    std::vector<int> counts(c->hk.ccap);
    if (cudaMemcpy(counts.data(), c->bufs.cellCount, 4 * counts.size(), cudaMemcpyDeviceToHost))
        return 6;
    long long counted = 0;
    for (int v : counts) counted += v;
    if (counted != st->count) return 6;  // it did get to the second barrier, and no further
    if (cudaMemset(c->bufs.run, 0, sizeof(RunSync))) return 7;  // the missing block's exit
    int at = usable_again(c, st, want);
    if (at) return 10 + at;

    // arrivals that say that some block gave up: every wait ends at once
    if (cb_load_state(c, st) || !set_arrivals(c, kRunGaveUp)) return 20;
    if (cb_search_neighbors(c) != CB_ERR_CUDA) return 21;
    if (!sync_is_clear(c)) return 22;
    at = usable_again(c, st, want);
    if (at) return 30 + at;
    cb_report rep;
    if (!set_arrivals(c, kRunGaveUp)) return 40;
    if (cb_integrate(c, 5, &rep) != CB_ERR_CUDA || rep.status != CB_ERR_CUDA) return 41;
    if (!sync_is_clear(c)) return 42;
    if (cb_integrate(c, 5, &rep) != CB_ERR_CUDA) return 43;  // until a new state is loaded
    at = usable_again(c, st, want);
    if (at) return 50 + at;
    cudaFree(dmap);
    cudaFree(dbufs);
    return cb_destroy(c) ? 60 : 0;
}
