// Levels of one graph in the shared memory of one block.
//
// A level pass over a deep graph is one hop per level, and its time is the
// hop's latency.  Through L2 a hop takes 1.8 us (a published word has to
// reach L2 and a poll to come back): the 64x64 multiplier's 501 levels 0.92
// ms, three times in one `rw; st`.  A graph of up to 57,000 nodes has its
// words in one block's shared memory instead: the threads take the nodes in
// order, a row at a time, and poll their two fanins' words there.  The polls
// of waiting warps bound the hop: 512 threads are faster than 1,024 (those
// 501 levels 0.13 ms against 0.16), and so is one node a thread than two or
// four (0.14, 0.17).  That is in level order, as the deduplication and `st` have
// it; in the multiplier's own order, the front's, a row waits on more of its
// own nodes: 0.48 ms, 0.54 through L2.
#include "levels.cuh"

namespace culs {

namespace {

constexpr int kLevelsThreads = 512;
constexpr int kUnresolved = -1;  // word of a node whose fanins are not all known; 0: pending, else 2 * level + phase + 1

// Every warp takes its rows in order and waits only for nodes earlier in the
// order, whose rows other warps take at the same time or took before, so the
// waits end; they are bounded all the same.  A fanin later in the order that
// is not known yet leaves the node unresolved, and so does an unresolved
// fanin; such nodes are tried again, all together, until a round resolves
// none.
__global__ void __launch_bounds__(kLevelsThreads, 1) k_levels_block(LevelsArgs A) {
    extern __shared__ int s_word[];
    volatile int *word = s_word;
    const int tid = threadIdx.x, n = (int)A.n;
    for (int i = tid; i < n; i += kLevelsThreads) s_word[i] = 0;
    __syncthreads();
    const int64_t lim = spin_limit(A.status);
    int top = 0, open = 0;
    auto load = [&](int i, int &a, int &b) {
        a = kLevelSkip, b = 0;
        if (i < n) {
            a = A.a0[i];
            b = A.a1[i];
            if (A.pre && A.pre[i] != -1) a = kLevelZero;
        }
    };
    auto settle = [&](int i, int a, int b, int x0, int x1) {
        const int e0 = x0 - 1, e1 = x1 - 1;
        const int lv = 1 + max(e0 >> 1, e1 >> 1);
        const int v = 2 * lv + (((e0 ^ a) & (e1 ^ b)) & 1);
        word[i] = v + 1;
        const int to = A.posOf ? A.posOf[i] : i;
        if (A.level) A.level[to] = lv;
        if (A.levelPhase) A.levelPhase[to] = v;
        if (!A.counted || A.counted[to]) top = max(top, lv);
    };
    int na, nb;
    load(tid, na, nb);
    for (int row = 0; row < n; row += kLevelsThreads) {
        const int i = row + tid;
        const int a = na, b = nb;
        load(i + kLevelsThreads, na, nb);  // the next row's, while this one waits
        if (a == kLevelZero) word[i] = 1;
        bool pend = a >= 0;
        const int u0 = a >> 1, u1 = b >> 1;
        for (int64_t it = 0; __any_sync(0xffffffffu, pend); it++) {
            if (pend) {
                const int x0 = word[u0], x1 = word[u1];
                const bool later0 = x0 == 0 && u0 >= i, later1 = x1 == 0 && u1 >= i;
                if (x0 > 0 && x1 > 0) {
                    settle(i, a, b, x0, x1);
                    pend = false;
                } else if (x0 == kUnresolved || x1 == kUnresolved || later0 || later1) {
                    word[i] = kUnresolved;
                    open++;
                    pend = false;
                } else if (it >= lim) {
                    set_status(A.status, kDevWaitTimeout);
                    word[i] = kUnresolved;
                    pend = false;
                }
            }
        }
    }
    while (__syncthreads_or(open)) {
        int got = 0;
        for (int i = tid; i < n && open; i += kLevelsThreads) {
            if (word[i] != kUnresolved) continue;
            int a, b;
            load(i, a, b);
            const int x0 = word[a >> 1], x1 = word[b >> 1];
            if (x0 <= 0 || x1 <= 0) continue;
            settle(i, a, b, x0, x1);
            open--;
            got = 1;
        }
        if (!__syncthreads_or(got)) break;
    }
    if (open && A.unsettled) atomicAdd(A.unsettled, open);
    top = __reduce_max_sync(0xffffffffu, top);
    if ((tid & 31) == 0 && top > 0) {
        if (A.depth0) atomicMax(A.depth0, top);
        if (A.depth1) atomicMax(A.depth1, top);
    }
}

}  // namespace

cudaError_t levels_block(const LevelsArgs &A, cudaStream_t s) {
    static_assert(kLevelsBlockMax * sizeof(int) <= 227 * 1024 - 1024, "shared memory of a block");
    const int smem = (int)(A.n * sizeof(int));
    const cudaError_t e =
        cudaFuncSetAttribute(k_levels_block, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kLevelsBlockMax * sizeof(int)));
    if (e != cudaSuccess) return e;
    k_levels_block<<<1, kLevelsThreads, smem, s>>>(A);
    return cudaGetLastError();
}

}  // namespace culs
