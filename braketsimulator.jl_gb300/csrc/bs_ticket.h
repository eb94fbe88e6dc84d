// The host's wait for a result that a kernel writes into mapped host memory, followed by a ticket.
#pragma once
#include <atomic>
#include <chrono>
#include <cstdint>
#include "../../include/braket_gb300.h"

// Polls the word for the ticket for `seconds`, then calls sync (which waits for the stream and returns its status).
// Only a ticket that is there stands for a result: BS_ERR_TIMEOUT where the stream ended without it.
template <typename Sync>
int bs_poll_ticket(const volatile int64_t* word, int64_t ticket, double seconds, Sync sync) {
    const auto t0 = std::chrono::steady_clock::now();
    for (uint32_t it = 0; *word != ticket; it++)
        if ((it & 1023u) == 1023u && std::chrono::steady_clock::now() - t0 > std::chrono::duration<double>(seconds)) {
            const int rc = sync();
            if (rc) return rc;
            if (*word != ticket) return BS_ERR_TIMEOUT;
            break;
        }
    std::atomic_thread_fence(std::memory_order_acquire);
    return BS_OK;
}
