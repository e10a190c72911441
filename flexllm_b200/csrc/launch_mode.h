// How the kernels that this thread launches follow the ones in front of them (host code only).
//
// Programmatic dependent launch: kernels carry the stream-serialization attribute, so that a kernel's launch and the start of its CTAs overlap the
// tail of the kernel in front. Every kernel launched that way lets its own dependents start (pdl_launch) and waits until the kernel in front has
// completed and flushed (pdl_wait) before it touches memory that is written in its stream.
#pragma once

namespace flexllm {

enum LaunchMode {
    kWhole = 0,         // every kernel starts behind the whole one before
    // A chain of launches. Its first kernel either carries no attribute (kChainStart) or lets others start only when its own wait is over (the
    // MLP block's norm); so the kernels behind it start when everything before the chain has completed, and between pdl_launch and pdl_wait they may
    // read what no kernel of the chain writes.
    kChain,
    kChainStart,
    kSetUp,             // overlapped behind whatever is in front, nothing protected: a kernel may set itself up (barriers, TMEM, descriptors) and read nothing
};
extern thread_local LaunchMode g_pdl;
bool programmatic_launches();          // FLEXLLM_PDL=0 in the environment: kWhole throughout

inline bool in_chain() { return g_pdl == kChain || g_pdl == kChainStart; }
inline bool may_read_ahead() { return g_pdl == kChain; }                             // of the next kernel
inline bool programmatic_next() { return g_pdl == kChain || g_pdl == kSetUp; }       // whether the next kernel carries the attribute
inline void launched() { if (g_pdl == kChainStart) g_pdl = kChain; }

// Launches in its scope are set up under the tail of whatever is in front, also outside a chain. A kernel that holds TMEM lets others start only once
// it has taken its columns. Product of 128 x 2048 x 2048, calls in a row: 8.2 -> 6.7 us; 9 to 8192 rows of nine matrices 1.06 times as fast, of the
// small ones up to 1.19.
struct SetUpEarly {
    const bool set = g_pdl == kWhole && programmatic_launches();
    SetUpEarly() { if (set) g_pdl = kSetUp; }
    ~SetUpEarly() { if (set) g_pdl = kWhole; }
};
// Around the launches of kernels that read something before their wait: outside a chain they are launched whole.
struct ReadsAhead {
    const bool set = g_pdl == kSetUp;
    ReadsAhead() { if (set) g_pdl = kWhole; }
    ~ReadsAhead() { if (set) g_pdl = kSetUp; }
};

}  // namespace flexllm
