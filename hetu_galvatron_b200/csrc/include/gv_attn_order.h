// Which barrier says that a product of the attention forward kernel is finished. Plain C++: the kernel and the host-side check of
// its waits (sim/attention_order_sim.cpp) share it.
#ifndef GV_ATTN_ORDER_H
#define GV_ATTN_ORDER_H

namespace gv {

// An mbarrier only tells the parity of its completed phases, so a wait for phase n is sound where n or n + 1 phases can be
// complete and no other number. The product P V of block j completes phase j / 2 of barrier j % 2. Whoever waits for block k
// (the issuer before S of k + 2, the softmax in block k + 1 before it rescales O, and after its last block k) has S of block
// k + 1 or k behind it, which was issued after block k - 2 was finished; and block k + 2 cannot be multiplied while the
// waiting thread has not arrived with its P. With one barrier for all blocks the last wait could find k - 1, k or k + 1
// complete: a warp that was held up after handing over its last P missed the phase for good.
struct PvPhase { int barrier; unsigned parity; };
constexpr int PV_BARRIERS = 2;
constexpr PvPhase pv_phase(int block) { return {block & 1, static_cast<unsigned>(block >> 1) & 1u}; }

}  // namespace gv
#endif
