// The GPU that launch shapes are chosen for.
#pragma once

namespace whir {
namespace gpu {

constexpr int SMS = 152;  // GB300

}  // namespace gpu
}  // namespace whir
