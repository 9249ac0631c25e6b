// in_turn.hpp -- host control flow of calls that must be completed whatever one of them does.
#pragma once
#include <cstddef>
#include <exception>

namespace mf3d {

// f(0) .. f(n - 1), all of them; the first exception is thrown after the last call
template <class F> void each_then_throw(size_t n, F&& f) {
    std::exception_ptr first;
    for (size_t i = 0; i < n; ++i) {
        try {
            f(i);
        } catch (...) {
            if (!first) first = std::current_exception();
        }
    }
    if (first) std::rethrow_exception(first);
}

// f(), then after(failed) whether f threw or not; f's exception is thrown rather than one of after's
template <class F, class A> void then_always(F&& f, A&& after) {
    std::exception_ptr first;
    try {
        f();
    } catch (...) {
        first = std::current_exception();
    }
    try {
        after(first != nullptr);
    } catch (...) {
        if (!first) throw;
    }
    if (first) std::rethrow_exception(first);
}

} // namespace mf3d
