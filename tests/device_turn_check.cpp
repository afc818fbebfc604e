/* DeviceTurn against a device of its own: the runtime calls that it makes are
 * defined here, grids are threads that run for a while, and a grid that starts
 * beside another one or beside a stay is counted. Built and run by
 * test_device_turn.py; prints "ok" or what went wrong. */

#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <future>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "common.hpp"
#include "device_turn.hpp"

using namespace nemo_b200;
using std::chrono::microseconds;

/* a stream: the work queued on it so far; an event: the work it stands for */
struct CUstream_st { std::vector<std::shared_future<void>> queue; };
struct CUevent_st { std::vector<std::shared_future<void>> work; };

static std::atomic<int> g_grids{0}, g_stays{0}, g_overlaps{0}, g_ran{0};

static bool ready(const std::shared_future<void>& f) { return f.wait_for(microseconds(0)) == std::future_status::ready; }

extern "C" {
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = new CUevent_st; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { e->work = s->queue; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned)
{
	s->queue.insert(s->queue.end(), e->work.begin(), e->work.end());
	return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e)
{
	for(auto& f : e->work) if(!ready(f)) return cudaErrorNotReady;
	return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
}

namespace nemo_b200 {
void cudaCheck(int err, const char*, const char*, int) { if(err) abort(); }
}

/* a finite grid after everything queued on the stream */
static void
launch(cudaStream_t s, int us = 300)
{
	auto before = s->queue;
	auto f = std::async(std::launch::async, [before, us] {
		for(auto& b : before) b.wait();
		if(++g_grids != 1 || g_stays != 0) g_overlaps++;
		std::this_thread::sleep_for(microseconds(us));
		if(g_stays != 0) g_overlaps++;
		g_ran++;
		g_grids--;
	}).share();
	s->queue.assign(1, f);
}

/* A simulation stepped without a pause */
struct Owner : Stay {
	std::mutex lock;
	std::atomic<bool> on{false};
	int stays = 0, commands = 0, others = 0, ended = 0;

	void end() { if(on) { on = false; g_stays--; } }
	void endStay() noexcept override
	{
		std::lock_guard<std::mutex> guard(lock);
		ended += on ? 1 : 0;
		end();
	}
	void step()
	{
		if(on && DeviceTurn::wanted(0)->load() == 0) {
			std::lock_guard<std::mutex> guard(lock);
			if(on) {
				std::this_thread::sleep_for(microseconds(15));
				commands++;
				return;
			}
		}
		{
			std::lock_guard<std::mutex> guard(lock);
			end();
		}
		const bool stayed = DeviceTurn::tryStay(0, this, [this] {
			std::lock_guard<std::mutex> guard(lock);
			if(g_grids != 0) g_overlaps++;
			if(++g_stays != 1) g_overlaps++;
			on = true;
			stays++;
		});
		if(!stayed) {
			others++;   /* one launch whose blocks do not wait */
			std::this_thread::sleep_for(microseconds(15));
		}
	}
};

int
main()
{
	std::atomic<bool> stop{false};
	/* a hang is a failure */
	std::thread([] { std::this_thread::sleep_for(std::chrono::seconds(60)); printf("hung\n"); fflush(stdout); _Exit(1); }).detach();
	const int TURNS = 150;
	std::vector<std::thread> grids, steppers;
	Owner a, b;
	for(Owner* o : {&a, &b}) steppers.emplace_back([o, &stop] { while(!stop) o->step(); });
	for(int k = 0; k < 2; ++k) {
		grids.emplace_back([k] {
			CUstream_st s;
			for(int t = 0; t < TURNS; ++t) {
				{
					DeviceTurn turn(0, &s);
					launch(&s);
					if(t % 3 == 0) launch(&s);
				}
				if(t % 10 == 9) std::this_thread::sleep_for(std::chrono::milliseconds(2 + k));
			}
			for(auto& f : s.queue) f.wait();
		});
	}
	for(auto& t : grids) t.join();
	stop = true;
	for(auto& t : steppers) t.join();
	const int want = 2 * (TURNS + (TURNS + 2) / 3);
	std::string bad;
	if(g_overlaps) bad += "overlaps ";
	if(g_ran != want) bad += "grids lost ";
	if(a.stays + b.stays == 0 || a.others + b.others == 0) bad += "one way of stepping not taken ";
	/* nothing in flight: a stay starts, another owner's or a turn ends it;
	 * a grid in flight: none starts */
	a.end();
	b.end();
	a.ended = b.ended = 0;
	a.step();
	if(!a.on) bad += "no stay on an idle device ";
	b.step();
	if(a.on || a.ended != 1 || !b.on) bad += "two stays ";
	CUstream_st s;
	{ DeviceTurn turn(0, &s); }
	if(b.on || b.ended != 1) bad += "a stay beside a turn ";
	a.step();
	a.end();
	DeviceTurn::leave(0, &a);
	{ DeviceTurn turn(0, &s); }
	if(a.ended != 1) bad += "an owner that has left was called ";
	{
		DeviceTurn turn(0, &s);
		launch(&s, 200000);
		bool stayed = false;
		std::thread([&] { stayed = DeviceTurn::tryStay(0, &b, [] {}); }).join();
		if(stayed) bad += "a stay beside a held turn ";
	}
	if(DeviceTurn::tryStay(0, &b, [] {})) bad += "a stay beside a grid ";
	for(auto& f : s.queue) f.wait();
	printf("%s\n", bad.empty() ? "ok" : bad.c_str());
	fflush(stdout);
	_Exit(bad.empty() ? 0 : 1);
}
