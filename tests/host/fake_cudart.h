// Hooks of the fake CUDA runtime (fake_cudart.cpp).
#pragma once
#include <functional>

bool fake_capturing();
// runs a kernel's function, or records it while a stream is captured
void fake_launch(std::function<void()> kernel);
int& fake_graph_launches();
