// A few threads that copy memory in chunks beside the calling thread: what tie_cuda_moe_ffn moves between pageable
// host buffers and the pinned staging.  One owner (the context's calling thread) at a time.  Between the copies of a call
// (in, compute, out: waking a sleeping thread costs as much as copying a chunk) the helpers stay awake, for SPIN_US at most;
// when the call ends (rest) they sleep, so that the threads of a caller's own pool find the cores free.
#pragma once

#include <string.h>

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <mutex>
#include <thread>

namespace tie {

class CopyPool {
	static constexpr int MAX_CHUNKS = 64, MAX_HELPERS = 3, SPIN_US = 400;
	std::mutex mutex_;
	std::condition_variable wake_, idle_;
	std::thread helpers_[MAX_HELPERS];
	int n_helpers_ = 0, inside_ = 0;  // helpers inside the current job (under mutex_)
	std::atomic<uint64_t> job_{0};	  // (written under mutex_)
	std::atomic<bool> in_call_{false};
	bool open_ = false, quit_ = false;
	char *dst_ = nullptr;
	const char *src_ = nullptr;
	size_t bytes_ = 0, chunk_ = 0;
	int n_ = 0;
	std::atomic<int> next_{0}, allowed_{0}, left_{0};
	std::atomic<bool> done_[MAX_CHUNKS];

	void work()
	{
		uint64_t seen = 0;
		std::unique_lock<std::mutex> lk(mutex_);
		for (;;) {
			if (seen) {
				lk.unlock();
				const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(SPIN_US);
				while (in_call_.load(std::memory_order_relaxed) && job_.load(std::memory_order_acquire) == seen &&
				       std::chrono::steady_clock::now() < until)
					std::this_thread::yield();
				lk.lock();
			}
			wake_.wait(lk, [&] { return quit_ || (open_ && job_.load(std::memory_order_relaxed) != seen); });
			if (quit_)
				return;
			seen = job_.load(std::memory_order_relaxed);
			inside_++;
			lk.unlock();
			while (left_.load(std::memory_order_acquire) > 0)
				if (!step())
					std::this_thread::yield();  // (the next chunk has not arrived yet)
			lk.lock();
			if (--inside_ == 0)
				idle_.notify_one();
		}
	}

public:
	CopyPool()
	{
		const unsigned cores = std::thread::hardware_concurrency();
		const int want = cores > 1 ? (int)cores - 1 : 0;
		for (int i = 0; i < (want < MAX_HELPERS ? want : MAX_HELPERS); i++) {
			try {
				helpers_[i] = std::thread([this] { work(); });
			} catch (...) {	 // no thread to be had: the caller copies alone
				break;
			}
			n_helpers_++;
		}
	}
	~CopyPool()
	{
		{
			std::lock_guard<std::mutex> lk(mutex_);
			quit_ = true;
		}
		wake_.notify_all();
		for (int i = 0; i < n_helpers_; i++)
			helpers_[i].join();
	}
	CopyPool(const CopyPool &) = delete;
	CopyPool &operator=(const CopyPool &) = delete;

	// n chunks of `chunk` bytes (the last one shorter); the first `allowed` of them may be copied at once.
	void begin(char *dst, const char *src, size_t bytes, size_t chunk, int n, int allowed)
	{
		{
			std::lock_guard<std::mutex> lk(mutex_);
			dst_ = dst;
			src_ = src;
			bytes_ = bytes;
			chunk_ = chunk;
			n_ = n;
			for (int i = 0; i < n; i++)
				done_[i].store(false, std::memory_order_relaxed);
			next_.store(0, std::memory_order_relaxed);
			allowed_.store(allowed, std::memory_order_relaxed);
			left_.store(n, std::memory_order_release);
			open_ = true;
			in_call_.store(true, std::memory_order_relaxed);
			job_.fetch_add(1, std::memory_order_release);
		}
		wake_.notify_all();
	}
	// The call that copied is over.
	void rest() { in_call_.store(false, std::memory_order_relaxed); }
	void allow(int n) { allowed_.store(n, std::memory_order_release); }
	bool done(int i) const { return done_[i].load(std::memory_order_acquire); }
	// Copies one chunk if there is one to copy.
	bool step()
	{
		int i = next_.load(std::memory_order_relaxed);
		do {
			if (i >= allowed_.load(std::memory_order_acquire))
				return false;
		} while (!next_.compare_exchange_weak(i, i + 1, std::memory_order_relaxed));
		const size_t o = (size_t)i * chunk_;
		memcpy(dst_ + o, src_ + o, o + chunk_ < bytes_ ? chunk_ : bytes_ - o);
		done_[i].store(true, std::memory_order_release);
		left_.fetch_sub(1, std::memory_order_acq_rel);
		return true;
	}
	// Every chunk that was handed out is copied and no helper is inside the job any more (chunks that were never
	// allowed are given up).
	void end()
	{
		const int never = n_ - allowed_.load(std::memory_order_relaxed);
		if (never > 0)
			left_.fetch_sub(never, std::memory_order_acq_rel);
		while (left_.load(std::memory_order_acquire) > 0)
			if (!step())
				std::this_thread::yield();
		std::unique_lock<std::mutex> lk(mutex_);
		open_ = false;
		idle_.wait(lk, [&] { return inside_ == 0; });
	}
};

}  // namespace tie
