// result_slots.h -- page-locked slots for the results of diagnostics calls,
// handed to handles out of blocks of kSlots: pinning costs the better part of
// a millisecond, and the server makes and frees handles at a high rate.
//
// A block belongs to the context that pinned it (told by its id) and dies with
// it (a device reset), so a slot is handed out only in that context and a
// block of another one is neither used nor freed.  A block whose slots have all
// come back is given back when it is not the context's last with room: what
// stays pinned is at most one empty block per context, and beyond that the
// blocks that handles still hold.  One lock guards the list; Mem::alloc and
// Mem::free run under it.
#pragma once
#include <stddef.h>
#include <mutex>
#include <new>

namespace scp {

struct SlotBlock;
struct ResultSlot {
    double *p;
    SlotBlock *block;
    ResultSlot *next;
};
struct SlotBlock {
    static constexpr int kSlots = 256;
    double *mem;
    unsigned long long ctx;
    int used;
    ResultSlot *free_list;
    SlotBlock *next;
    ResultSlot slot[kSlots];
};

// Mem: static double *alloc(size_t bytes) (null on failure), static void free(double *)
template <class Mem, int WORDS>
class SlotPool {
    std::mutex mu;
    SlotBlock *blocks = nullptr;

    SlotBlock *with_room(unsigned long long ctx, const SlotBlock *but) {
        for (SlotBlock *b = blocks; b; b = b->next)
            if (b != but && b->ctx == ctx && b->used < SlotBlock::kSlots) return b;
        return nullptr;
    }

public:
    ResultSlot *take(unsigned long long ctx) {
        std::lock_guard<std::mutex> lk(mu);
        SlotBlock *b = with_room(ctx, nullptr);
        if (!b) {
            double *p = Mem::alloc(sizeof(double) * WORDS * SlotBlock::kSlots);
            if (!p) return nullptr;
            b = new (std::nothrow) SlotBlock{p, ctx, 0, nullptr, blocks, {}};
            if (!b) {
                Mem::free(p);
                return nullptr;
            }
            for (int q = SlotBlock::kSlots - 1; q >= 0; q--) {
                b->slot[q] = ResultSlot{p + (size_t)q * WORDS, b, b->free_list};
                b->free_list = &b->slot[q];
            }
            blocks = b;
        }
        ResultSlot *r = b->free_list;
        b->free_list = r->next;
        b->used++;
        return r;
    }
    // ctx: the context current now
    void give(ResultSlot *r, unsigned long long ctx) {
        std::lock_guard<std::mutex> lk(mu);
        SlotBlock *b = r->block;
        r->next = b->free_list;
        b->free_list = r;
        if (--b->used || b->ctx != ctx || !with_room(ctx, b)) return;
        for (SlotBlock **at = &blocks; *at; at = &(*at)->next)
            if (*at == b) {
                *at = b->next;
                break;
            }
        Mem::free(b->mem);
        delete b;
    }
};

}  // namespace scp
