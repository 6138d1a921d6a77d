// Runs segmentctscans_b200/csrc/block.cuh on the host: the threads of a block as coroutines that
// advance one at a time, each until it waits for others at a barrier or a warp instruction, the
// runnable thread of the highest rank first.  A warp at the front therefore runs as far ahead of
// the others as the barriers let it, which is where a value that is read behind a barrier and written
// by a thread that has gone on shows; the ranks are also drawn at random.  Threads that wait at a
// barrier when another has ended count as an error.
#include <ucontext.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#define __device__
#define __forceinline__ inline

namespace {

enum class At { kRun, kBarrier, kWarp, kDone };
struct Thread {
    ucontext_t uc;
    std::vector<char> stack;
    At at = At::kRun;
    int rank = 0;
    unsigned in = 0, out = 0;  // this thread's value for a barrier or warp instruction, and the result
    int src = 0;               // shuffle: the source lane, -1 for a ballot
};
struct Dim {
    unsigned x;
};
constexpr int kThreads = 256;
std::vector<Thread> threads(kThreads);
ucontext_t scheduler;
int current = 0;
Dim threadIdx{0};

unsigned wait_at(At at, unsigned in, int src)
{
    Thread &t = threads[(size_t)current];
    t.at = at;
    t.in = in;
    t.src = src;
    swapcontext(&t.uc, &scheduler);
    return t.out;
}
void __syncthreads() { wait_at(At::kBarrier, 0, 0); }
int __syncthreads_count(int p) { return (int)wait_at(At::kBarrier, p != 0, 0); }
int __syncthreads_or(int p) { return wait_at(At::kBarrier, p != 0, 0) != 0; }
unsigned __ballot_sync(unsigned, int p) { return wait_at(At::kWarp, p != 0, -1); }
int __shfl_sync(unsigned, int v, int src) { return (int)wait_at(At::kWarp, (unsigned)v, src); }
int __popc(unsigned v) { return __builtin_popcount(v); }
int atomicAdd(int *p, int v)
{
    const int old = *p;
    *p += v;
    return old;
}

}  // namespace

#include "block.cuh"

namespace {

void (*body)();
void entry()
{
    body();
    threads[(size_t)current].at = At::kDone;
    swapcontext(&threads[(size_t)current].uc, &scheduler);
}

// Runs f in every thread; false when threads wait for one another for ever.
bool run_block(void (*f)(), const std::vector<int> &rank)
{
    body = f;
    for (int i = 0; i < kThreads; ++i) {
        Thread &t = threads[(size_t)i];
        t.stack.resize(64 << 10);
        t.at = At::kRun;
        t.rank = rank[(size_t)i];
        getcontext(&t.uc);
        t.uc.uc_stack.ss_sp = t.stack.data();
        t.uc.uc_stack.ss_size = t.stack.size();
        t.uc.uc_link = nullptr;
        makecontext(&t.uc, entry, 0);
    }
    while (true) {
        int next = -1, done = 0, waiting = 0;
        for (int i = 0; i < kThreads; ++i) {
            const Thread &t = threads[(size_t)i];
            if (t.at == At::kRun && (next < 0 || t.rank < threads[(size_t)next].rank)) next = i;
            done += t.at == At::kDone;
            waiting += t.at == At::kBarrier;
        }
        if (next >= 0) {
            current = next;
            threadIdx.x = (unsigned)next;
            swapcontext(&scheduler, &threads[(size_t)next].uc);
            // a warp whose 32 lanes have all arrived goes on
            const int w = next / 32 * 32;
            bool all = true;
            for (int i = w; i < w + 32; ++i) all = all && threads[(size_t)i].at == At::kWarp;
            if (all) {
                unsigned ballot = 0;
                for (int i = 0; i < 32; ++i) ballot |= (threads[(size_t)(w + i)].in & 1u) << i;
                for (int i = w; i < w + 32; ++i) {
                    Thread &t = threads[(size_t)i];
                    t.out = t.src < 0 ? ballot : threads[(size_t)(w + t.src)].in;
                }
                for (int i = w; i < w + 32; ++i) threads[(size_t)i].at = At::kRun;
            }
            continue;
        }
        if (done == kThreads) return true;
        if (waiting != kThreads) return false;  // some have ended, or wait elsewhere
        unsigned sum = 0;
        for (const Thread &t : threads) sum += t.in;
        for (Thread &t : threads) t.out = sum, t.at = At::kRun;
    }
}

// ---- LoopList: every voxel that needs the loop is run once, with the values that were put in
constexpr int kMaxChunks = potts::kLoopChunks;
double share[kMaxChunks];  // share of the voxels that need the loop, per chunk
std::vector<char> wanted;
std::vector<int> ran;
bool wrong_values = false;

template <int N>
struct Shared {
    static potts::LoopList<N> list;
};
template <int N>
potts::LoopList<N> Shared<N>::list;

template <int N>
void list_kernel()
{
    auto &list = Shared<N>::list;
    if (threadIdx.x == 0) list.count = 0;
    __syncthreads();
    int n = 0;
    for (int c = 0; c < potts::kLoopChunks; ++c) {
        const int64_t o = (int64_t)c * kThreads + threadIdx.x;
        const bool need = wanted[(size_t)o] != 0;
        const int e = list.add(need);
        if (need && (e < 0 || e >= potts::LoopList<N>::kCap)) {
            wrong_values = true;
        } else if (need) {
            for (int j = 0; j < N; ++j) list.v[j][e] = (float)(o * 64 + j);
            list.off[e] = o;
        }
        list.flush(n, need, c + 1 == potts::kLoopChunks, [&](int i) {
            const int64_t p = list.off[i];
            if (p < 0 || p >= (int64_t)ran.size()) {
                wrong_values = true;
                return;
            }
            ++ran[(size_t)p];
            for (int j = 0; j < N; ++j) wrong_values = wrong_values || list.v[j][i] != (float)(p * 64 + j);
        });
    }
}

template <int N>
bool check_list(const std::vector<int> &rank, std::mt19937 &rng)
{
    wanted.assign((size_t)kMaxChunks * kThreads, 0);
    ran.assign(wanted.size(), 0);
    wrong_values = false;
    for (int c = 0; c < kMaxChunks; ++c)
        for (int i = 0; i < kThreads; ++i)
            wanted[(size_t)(c * kThreads + i)] = std::uniform_real_distribution<double>(0.0, 1.0)(rng) < share[c];
    for (auto &o : Shared<N>::list.off) o = -1;
    if (!run_block(list_kernel<N>, rank) || wrong_values) return false;
    for (size_t i = 0; i < ran.size(); ++i)
        if (ran[i] != wanted[i]) return false;
    return true;
}

// ---- sync_aborted: when one warp's wait gives up, all leave the loop after the same pass
volatile int abort_flag = 0;
int give_up_warp = 0, give_up_pass = 0;
std::vector<int> passes;

void abort_kernel()
{
    if (threadIdx.x == 0) abort_flag = 0;
    __syncthreads();
    int pass = 0;
    for (; pass < 6; ++pass) {
        if ((int)threadIdx.x / 32 == give_up_warp && pass == give_up_pass) abort_flag = 1;
        if (potts::sync_aborted(&abort_flag)) break;
    }
    passes[threadIdx.x] = pass;
    __syncthreads();
}

bool check_abort(const std::vector<int> &rank)
{
    for (give_up_warp = 0; give_up_warp < kThreads / 32; ++give_up_warp)
        for (give_up_pass = 0; give_up_pass <= 6; ++give_up_pass) {  // 6: none
            passes.assign((size_t)kThreads, -1);
            if (!run_block(abort_kernel, rank)) return false;
            for (int p : passes)
                if (p != give_up_pass) return false;
        }
    return true;
}

}  // namespace

int main()
{
    std::mt19937 rng(1);
    // first warp first, last warp first, warps and then single threads at random
    std::vector<std::vector<int>> ranks;
    for (int k = 0; k < 6; ++k) {
        std::vector<int> r((size_t)kThreads), w(8);
        for (int i = 0; i < 8; ++i) w[(size_t)i] = k == 1 ? 7 - i : i;
        if (k > 1) std::shuffle(w.begin(), w.end(), rng);
        for (int i = 0; i < kThreads; ++i) r[(size_t)i] = w[(size_t)(i / 32)] * 32 + i % 32;
        if (k > 3) std::shuffle(r.begin(), r.end(), rng);
        ranks.push_back(r);
    }
    // shares of voxels that need the loop: none, few, about the threshold of a flush, all; and chunks of
    // unlike shares, the last ones empty as past the end of the volume
    const double shares[][4] = {{0, 0, 0, 0},       {0.004, 0.004, 0.004, 0.004}, {0.13, 0.13, 0.13, 0.13},
                                {0.5, 0.5, 0.5, 0.5}, {1, 1, 1, 1},                {1, 0, 1, 0},
                                {0, 1, 0.02, 0},     {0.3, 0.9, 0, 0},            {1, 0.004, 0, 0}};
    int bad = 0;
    for (const auto &s : shares)
        for (const auto &r : ranks) {
            for (int c = 0; c < kMaxChunks; ++c) share[c] = s[c];
            // 512 entries (K = 2 .. 6 forward, K = 2, 3 adjoint) and 256 (adjoint of K >= 4)
            bad += !check_list<6>(r, rng) + !check_list<18>(r, rng) + !check_list<21>(r, rng) + !check_list<33>(r, rng);
        }
    std::printf("loop list: %d of %zu runs wrong\n", bad, sizeof(shares) / sizeof(shares[0]) * ranks.size() * 4);
    int apart = 0;
    for (const auto &r : ranks) apart += !check_abort(r);
    std::printf("abort: %d of %zu orders wrong\n", apart, ranks.size());
    return bad + apart != 0;
}
