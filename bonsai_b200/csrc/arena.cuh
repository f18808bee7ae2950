// Where a fit's device arrays live: one allocation for arrays of one lifetime,
// from a pool that the device's planes hold.
#pragma once

#include "common.cuh"

#include <algorithm>
#include <cstddef>
#include <memory>
#include <mutex>
#include <utility>
#include <vector>

namespace bb
{

// The pool of one device. Mapping and unmapping memory takes 0.1 to several
// ms a call, and up to a second where other processes use the driver, so up
// to 1 GiB stays mapped between fits. Every plane that has been fitted holds
// the pool; the last one to go gives all of it back. (The CUDA pool beneath
// orders its blocks by stream and takes calls from any thread.)
class MemPool
{
  public:
    explicit MemPool(int device)
    {
        cudaMemPoolProps props{};
        props.allocType     = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id   = device;
        BB_CHECK(cudaMemPoolCreate(&pool_, &props));
        uint64_t keep = k_keep;
        BB_CHECK(cudaMemPoolSetAttribute(pool_, cudaMemPoolAttrReleaseThreshold, &keep));
    }
    ~MemPool()
    {
        cudaMemPoolDestroy(pool_);
    }
    MemPool(MemPool const &)            = delete;
    MemPool &operator=(MemPool const &) = delete;

    void *alloc(size_t bytes, cudaStream_t s)
    {
        void *p = nullptr;
        with_trim([&] { return cudaMallocFromPoolAsync(&p, bytes, pool_, s); },
                  "cudaMallocFromPoolAsync");
        return p;
    }

    // The device's pool, made by its first holder.
    static std::shared_ptr<MemPool> of(int device)
    {
        Registry                   &r = registry();
        std::lock_guard<std::mutex> lock(r.mu);
        r.pools.resize(std::max(r.pools.size(), static_cast<size_t>(device) + 1));
        std::shared_ptr<MemPool> p = r.pools[device].lock();
        if (p == nullptr)
        {
            p               = std::make_shared<MemPool>(device);
            r.pools[device] = p;
        }
        return p;
    }

    // Runs an allocation; where it finds no memory, once more without the
    // pools' idle blocks.
    template <typename F> static void with_trim(F const &allocate, char const *what)
    {
        cudaError_t e = allocate();
        if (e == cudaErrorMemoryAllocation)
        {
            cudaGetLastError();
            Registry                             &r = registry();
            std::vector<std::shared_ptr<MemPool>> live;
            {
                std::lock_guard<std::mutex> lock(r.mu);
                for (std::weak_ptr<MemPool> const &w : r.pools)
                {
                    live.push_back(w.lock());
                }
            }
            for (std::shared_ptr<MemPool> const &p : live)
            {
                if (p != nullptr)
                {
                    cudaMemPoolTrimTo(p->pool_, 0);
                }
            }
            e = allocate();
        }
        check(e, what);
    }

  private:
    struct Registry
    {
        std::mutex                          mu;
        std::vector<std::weak_ptr<MemPool>> pools; // by device
    };
    static Registry &registry()
    {
        static Registry r;
        return r;
    }

    static constexpr uint64_t k_keep = uint64_t{1} << 30;
    cudaMemPool_t             pool_{};
};

// want() notes an array, alloc() makes one allocation for all of them and sets
// their pointers. A booster holds about seventy arrays, most of a few KB;
// allocated one by one, 64 boosters of 1,000 to 200,000 rows took 290 ms to
// create and 35 to close, and take 24 and 12; 7 class lanes of 581,012 rows
// 10-34 and 5-260, and take 3.3 and 1.3.
class Arena
{
  public:
    Arena() = default;
    ~Arena()
    {
        release();
    }
    Arena(Arena const &)            = delete;
    Arena &operator=(Arena const &) = delete;

    template <typename T, typename P> void want(P *&p, size_t n)
    {
        wanted_.emplace_back(reinterpret_cast<void **>(&p), bytes_);
        bytes_ += (std::max<size_t>(1, n) * sizeof(T) + k_align - 1) / k_align * k_align;
    }
    void alloc(std::shared_ptr<MemPool> pool, cudaStream_t s)
    {
        base_   = pool->alloc(bytes_, s);
        pool_   = std::move(pool);
        stream_ = s;
        for (auto const &[p, at] : wanted_)
        {
            *p = static_cast<char *>(base_) + at;
        }
        wanted_.clear();
    }
    // Frees on the stream it was allocated on; every other stream's use of the
    // arrays has to be over.
    void release()
    {
        if (base_ != nullptr)
        {
            cudaFreeAsync(base_, stream_);
            base_ = nullptr;
            pool_.reset();
        }
    }

  private:
    static constexpr size_t                 k_align = 256;
    std::vector<std::pair<void **, size_t>> wanted_;
    size_t                                  bytes_  = 0;
    void                                   *base_   = nullptr;
    cudaStream_t                            stream_ = nullptr;
    std::shared_ptr<MemPool>                pool_;
};

} // namespace bb
