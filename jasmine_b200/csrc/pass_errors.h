// Status of a pass from the error words that its last kernels copied beside its results (the device's word as each of them found it).
#pragma once
#include <cstdint>

namespace jsm {

// check(): reads the device's word, reports it and clears it.  The word belongs to all models of the device, so another caller may have read and
// cleared it since the copy: then the copied code stands (fail).  Status 0 is success.
template <typename Check, typename Fail>
inline auto pass_status(const int32_t* words, int n, Check check, Fail fail) -> decltype(check()) {
    int32_t code = 0;
    for (int i = 0; i < n && code == 0; ++i) code = words[i];
    if (code == 0) return decltype(check()){};
    const auto s = check();
    return s != decltype(check()){} ? s : fail(code);
}

}  // namespace jsm
