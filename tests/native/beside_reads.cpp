// What a kernel launched beside another reads from memory has no load but one past L1
// (dm_jobs.cuh compiled for the CPU): the jobs' inputs are of the type that sees to it,
// which converts to no pointer that could be read otherwise.
#include <type_traits>

#include "dm_jobs.cuh"

using namespace dm;

template <class F, class T>
constexpr bool past_l1 = std::is_same_v<F, PastL1<T>> && !std::is_convertible_v<F, const T*> &&
                         !std::is_convertible_v<F, const void*> && std::is_trivially_copyable_v<F>;

static_assert(past_l1<decltype(UnpackJob::file), uint8_t>);
static_assert(past_l1<decltype(FinishJobX::expect), uint4>);
static_assert(past_l1<decltype(TailJob::m), uint4>);
static_assert(past_l1<decltype(TailJob::g), uint4>);
static_assert(past_l1<decltype(TailJob::c), uint4>);
static_assert(past_l1<decltype(TailJob::l), uint4>);
static_assert(past_l1<decltype(TailJob::r), uint4>);
static_assert(past_l1<decltype(TailJob::file_id), uint32_t>);
// kernel parameters hold them as the bare pointer
static_assert(sizeof(PastL1<uint4>) == sizeof(void*));

int main() { return 0; }
