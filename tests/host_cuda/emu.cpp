// The fibers, barriers and launches behind cuda_runtime.h (see there), and entry points for the tests.
#include "cuda_runtime.h"

EmuIdx threadIdx, blockIdx, blockDim, gridDim;
long emu_mallocs = 0, emu_copies = 0;

// saves the callee-saved registers, leaves the stack pointer in *from and continues at to
extern "C" void emu_switch(void** from, void* to);
__asm__(
    ".text\n.globl emu_switch\nemu_switch:\n"
    "push %rbx\npush %rbp\npush %r12\npush %r13\npush %r14\npush %r15\n"
    "mov %rsp,(%rdi)\nmov %rsi,%rsp\n"
    "pop %r15\npop %r14\npop %r13\npop %r12\npop %rbp\npop %rbx\nret\n");

namespace emu {

constexpr size_t kStack = 192 << 10;
Fiber* cur = nullptr;
std::vector<int> order;
bool keep = false;

namespace {
struct Warp { Meet meet; uint64_t slot[2][32]; unsigned gen[32]; };
struct Block { std::vector<Warp> warps; Meet bar[16]; std::vector<double> smem; int index; };
std::vector<Block> blocks;
std::vector<Fiber> fibers;
std::vector<char*> stacks;
Meet cluster_meet;
const std::function<void()>* body;
void* main_sp;
int nthreads;

Warp& warp() { return blocks[cur->block].warps[cur->tid >> 5]; }
void yield() { emu_switch(&cur->sp, main_sp); }
void entry() {
    (*body)();
    cur->done = true;
    cur->ready = false;
    yield();
}
void resume(Fiber& f) {
    cur = &f;
    threadIdx = {(unsigned)f.tid, 0, 0};
    blockIdx = {(unsigned)blocks[f.block].index, 0, 0};
    emu_switch(&main_sp, f.sp);
}
}  // namespace

int block_threads() { return nthreads; }
int cluster_size() { return (int)blocks.size(); }
Meet& barrier(int id) { return blocks[cur->block].bar[id]; }
Meet& cluster_barrier() { return cluster_meet; }
double* dyn_smem() { return blocks[cur->block].smem.data(); }
double* dyn_smem_of(int rank) { return blocks[rank].smem.data(); }

void meet(Meet& m, int n, bool) {
    if (++m.arrived < n) {
        m.waiting.push_back(cur);
        cur->ready = false;
        yield();
        return;
    }
    for (Fiber* f : m.waiting) f->ready = true;
    m.waiting.clear();
    m.arrived = 0;
}
uint64_t* warp_slots() { return warp().slot[warp().gen[cur->tid & 31]++ & 1]; }
void warp_wait() { meet(warp().meet, 32); }

void launch(dim3 grid, dim3 block, size_t smem, const std::function<void()>& fn, int cluster) {
    nthreads = (int)block.x;
    const int nw = (nthreads + 31) / 32;
    gridDim = {grid.x, 1, 1};
    blockDim = {block.x, 1, 1};
    body = &fn;
    for (unsigned b0 = 0; b0 < grid.x; b0 += cluster) {
        blocks.assign(cluster, Block{});
        cluster_meet = Meet{};
        fibers.assign((size_t)cluster * nthreads, Fiber{});
        for (int c = 0; c < cluster; ++c) {
            Block& B = blocks[c];
            B.index = (int)b0 + c;
            B.warps.resize(nw);
            for (Warp& w : B.warps) std::memset(w.gen, 0, sizeof w.gen);
            B.smem.assign((smem + kGuard) / sizeof(double) + 1, std::nan(""));      // shared memory starts undefined
            std::memset((char*)B.smem.data() + smem, kGuardByte, kGuard);
        }
        for (size_t i = 0; i < fibers.size(); ++i) {
            if (stacks.size() <= i) stacks.push_back((char*)std::aligned_alloc(64, kStack));
            Fiber& f = fibers[i];
            f.tid = (int)(i % nthreads);
            f.block = (int)(i / nthreads);
            void** sp = (void**)(stacks[i] + kStack - 64);
            *--sp = nullptr;                                            // entry's return address (never used)
            *--sp = (void*)entry;
            for (int r = 0; r < 6; ++r) *--sp = nullptr;
            f.sp = sp;
        }
        std::vector<int> seq;                                           // warps of the cluster, in resuming order
        for (int w : order)
            for (int c = 0; c < cluster; ++c)
                if (w < nw) seq.push_back(c * nw + w);
        for (int w = 0; w < cluster * nw; ++w)
            if (std::find(seq.begin(), seq.end(), w) == seq.end()) seq.push_back(w);
        for (;;) {
            bool any = false;
            for (int w : seq) {
                bool ran = false;
                for (int l = 0; l < 32; ++l) {
                    const int t = (w % nw) * 32 + l;
                    if (t >= nthreads) break;
                    Fiber& f = fibers[(size_t)(w / nw) * nthreads + t];
                    if (f.ready) { resume(f); ran = true; }
                }
                any = any || ran;
                if (ran && keep) break;
            }
            if (!any) break;
        }
        for (const Block& B : blocks) check_guard((const unsigned char*)B.smem.data() + smem, "behind shared memory");
        for (const Fiber& f : fibers)
            if (!f.done) {
                std::fprintf(stderr, "emu: thread %d of block %d waits for ever\n", f.tid, (int)b0 + f.block);
                std::abort();
            }
    }
}

}  // namespace emu

// the resuming order of the warps of the launches that follow; keep: see emu::keep
extern "C" void emu_schedule(const int* warps, int n, int keep) {
    emu::order.assign(warps, warps + n);
    emu::keep = keep != 0;
}
extern "C" void emu_counts(long* mallocs, long* copies) {
    *mallocs = emu_mallocs;
    *copies = emu_copies;
}

// The deposit into compact beam sources of m = 0 runs (a pipelined run's rings), which no entry point calls by itself.
// cols: 7 columns of n; scale: null, or 1 / quantum per node for the exact format of two limbs of s_bits
#include "qz_internal.h"
extern "C" int emu_deposit_compact(int M, const double* r, const double* inv_h, const double* inv_V, double xi_min,
                                   double dxi, int K, int ngp, double* cols, long n, double q, const double* scale,
                                   int s_bits, double* bsrc) {
    qzb::BeamArgs B{};
    B.x = cols; B.y = cols + n; B.px = cols + 2 * n; B.py = cols + 3 * n; B.pz = cols + 4 * n; B.xi = cols + 5 * n;
    B.w = cols + 6 * n;
    B.n = n; B.q = q; B.m = 1.0;
    B.M = M; B.N = M - 1; B.R = r[M - 1];
    B.r = r; B.inv_h = inv_h; B.inv_V = inv_V;
    B.xi_min = xi_min; B.dxi = dxi; B.idxi = 1.0 / dxi; B.K = K; B.ngp = ngp;
    B.fx_scale = scale; B.fx_2s = std::ldexp(1.0, s_bits); B.fx_inv2s = std::ldexp(1.0, -s_bits);
    B.compact = 1;
    return (int)qzb::launch_beam_deposit(B, bsrc, nullptr);
}
