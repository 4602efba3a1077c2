// One element of a folded codeword: v0 + (r - x0) (v1 - v0) w for the pair (v0, v1) and its table entry (x0, w).
#pragma once
#include "gl_field.cuh"

namespace mb {
namespace bf {

GLF gl::E2 fold_pair_base(ulonglong2 v, ulonglong2 e, gl::E2 r) {
    const uint64_t dw = gl::mul(gl::sub(v.y, v.x), e.y);
    return gl::e2_canon(gl::E2{gl::mul_add(gl::sub(r.c0, e.x), dw, v.x), gl::mul(r.c1, dw)});
}
// r1w = 7 r.c1 mod p
GLF gl::E2 fold_pair_ext(gl::E2 v0, gl::E2 v1, ulonglong2 e, gl::E2 r, uint64_t r1w) {
    const gl::E2 dw = gl::e2_mul_base(gl::e2_sub(v1, v0), e.y);
    return gl::e2_canon(gl::e2_fma_pre(gl::E2Pre{gl::sub(r.c0, e.x), r.c1, r1w}, dw, v0));
}

}  // namespace bf
}  // namespace mb
